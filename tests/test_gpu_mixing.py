"""The one-launch Broyden step on the GPU against the update written out in numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(maps, steps, fraction):
    """Inputs of Broyden's second method (scalar 1) for n_out = maps(n_in, step)."""
    n, prev, F, V, W, out = 0.0, 0.0, 0.0, [], [], []
    for k in range(steps):
        Fc = n - maps(n, k)
        dF, F = Fc - F, Fc
        if k > 0:
            acc = sum(((v @ dF) * w for v, w in zip(V, W)), np.zeros_like(F))
            V.append(dF / (dF @ dF))
            W.append(-fraction * dF + (n - prev) - acc)
        acc = sum(((v @ F) * w for v, w in zip(V, W)), np.zeros_like(F))
        prev, n = n, n - fraction * F - acc
        out.append((n, np.abs(F).max()))
    return out


@pytest.mark.parametrize("S", [1, 7, 9, 511, 4097, 16384, 16385])
@pytest.mark.parametrize("device", [False, True])
def test_broyden_step_forms(S, device):
    """Fewer sites than the cluster has blocks, ragged pieces, both sides of the
    line to the general path.  Random maps: sums of S products, 1e-16 sqrt(S)
    each, amplified by at most 1e3 over six steps: 1e-11."""
    import torch
    from electrostatic_b200.negf import Broyden
    from electrostatic_b200.scf import device_view
    rng = np.random.default_rng(S)
    a, b = 0.5 + 0.2 * rng.random(S), rng.standard_normal(S)

    def maps(n, k):
        return a * n + b * (1.0 + 0.1 * k)

    steps = 6 if S > 1 else 1
    ref = _reference(maps, steps, 0.2)
    br = Broyden(torch.zeros(S, dtype=torch.float64, device="cuda"), max_step=20, fraction=0.2)
    view = device_view(br.input_device_ptr(), S)
    flags = torch.zeros(4, dtype=torch.int32, device="cuda")
    for k, (n, norm) in enumerate(ref):
        out = torch.from_numpy(np.ascontiguousarray(maps(view.cpu().numpy(), k))).cuda()
        if device:
            br.step_device(out, 1e-30, flags)
        else:
            assert abs(br.step(out) - norm) <= 1e-11 * abs(norm) + 1e-13
        torch.cuda.synchronize()
        got = view.cpu().numpy()
        assert np.abs(got - n).max() <= 1e-11 * np.abs(n).max(), k
    if device:
        assert flags.cpu().tolist() == [0, steps, 0, 0] and br.step_number == steps + 1
