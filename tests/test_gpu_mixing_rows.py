"""Broyden steps with a long history."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _time(S, rows):
    """A device-resident step at `rows` rows."""
    import torch
    from electrostatic_b200.negf import Broyden
    br = Broyden(torch.zeros(S, dtype=torch.float64, device="cuda"), max_step=rows + 60, fraction=0.1)
    flags = torch.zeros(4, dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(S)
    outs = [torch.randn(S, dtype=torch.float64, device="cuda", generator=g) for _ in range(8)]
    for k in range(rows):
        br.step_device(outs[k % 8], 1e-300, flags)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    ev[0].record()
    for k in range(30):
        br.step_device(outs[k % 8], 1e-300, flags)
    ev[1].record()
    torch.cuda.synchronize()
    assert flags.cpu().tolist() == [0, rows + 30, 0, 0]
    return ev[0].elapsed_time(ev[1]) / 30


def test_long_histories_use_the_whole_gpu():
    """500 rows of 12000 sites cost less than 500 rows of 16400 (one cluster took
    twice the time of the whole GPU)."""
    small, large = _time(12000, 500), _time(16400, 500)
    assert small <= 0.9 * large, (small, large)


@pytest.mark.parametrize("S,max_step", [(8000, 409), (8000, 410), (16384, 200), (16384, 201)])
@pytest.mark.parametrize("device", [False, True])
def test_both_sides_of_the_line(S, max_step, device):
    """Steps at the last and first max_step of the two forms against the update
    written out in numpy (1e-11: see test_broyden_step_forms)."""
    import torch
    from electrostatic_b200.negf import Broyden
    from electrostatic_b200.scf import device_view
    from test_gpu_mixing import _reference
    rng = np.random.default_rng(S)
    a, b = 0.5 + 0.2 * rng.random(S), rng.standard_normal(S)

    def maps(n, k):
        return a * n + b * (1.0 + 0.1 * k)
    br = Broyden(torch.zeros(S, dtype=torch.float64, device="cuda"), max_step=max_step, fraction=0.2)
    view = device_view(br.input_device_ptr(), S)
    flags = torch.zeros(4, dtype=torch.int32, device="cuda")
    for k, (n, _) in enumerate(_reference(maps, 6, 0.2)):
        out = torch.from_numpy(np.ascontiguousarray(maps(view.cpu().numpy(), k))).cuda()
        if device:
            br.step_device(out, 1e-30, flags)
        else:
            br.step(out)
        torch.cuda.synchronize()
        assert np.abs(view.cpu().numpy() - n).max() <= 1e-11 * np.abs(n).max(), k
