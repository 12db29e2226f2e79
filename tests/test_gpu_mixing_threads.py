"""Independent Broyden mixers stepped by two threads at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 400


def _run(S, max_step, stream, out, errors):
    """STEPS device-resident steps of n_out = a n_in + b; the last input and the flags."""
    import torch
    from electrostatic_b200.negf import Broyden
    from electrostatic_b200.scf import device_view
    try:
        with torch.cuda.stream(stream):
            rng = np.random.default_rng(S)
            n_out = torch.from_numpy(rng.standard_normal(S)).cuda()
            br = Broyden(torch.zeros(S, dtype=torch.float64, device="cuda"), max_step=max_step, fraction=0.2,
                         stream=stream)
            flags = torch.zeros(4, dtype=torch.int32, device="cuda")
            view = device_view(br.input_device_ptr(), S)
            for k in range(STEPS):
                if k % 20 == 0:
                    br.reset(stream=stream)
                br.step_device(n_out, 1e-300, flags, stream=stream)
            stream.synchronize()
            out[S] = (view.cpu().numpy().copy(), flags.cpu().tolist())
    except Exception as e:  # noqa: BLE001 - reported by the test
        errors.append(e)


def test_mixers_of_different_sizes_in_two_threads():
    """Mixers whose steps need 61 KB and 1 KB of shared memory a block: the
    steps of one do not change what the other may use, and both end where they
    end alone (bitwise)."""
    import torch
    sizes = [(1800, 1800), (64, 30)]
    streams = [torch.cuda.Stream() for _ in sizes]
    alone, together, errors = {}, {}, []
    for (S, m), s in zip(sizes, streams):
        _run(S, m, s, alone, errors)
    assert not errors, errors
    threads = [threading.Thread(target=_run, args=(S, m, s, together, errors)) for (S, m), s in zip(sizes, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for S, _ in sizes:
        assert np.array_equal(alone[S][0], together[S][0]) and alone[S][1] == together[S][1]


def test_launches_of_four_mixers_at_once():
    """8000 launches of one large and three small mixers, whose kernels return at
    once (skip word set), so that the host's calls meet as often as they can."""
    import torch
    errors = []

    def launch(S, max_step, stream):
        from electrostatic_b200.negf import Broyden
        try:
            with torch.cuda.stream(stream):
                out = torch.zeros(S, dtype=torch.float64, device="cuda")
                flags = torch.ones(8, dtype=torch.int32, device="cuda")
                br = Broyden(torch.zeros(S, dtype=torch.float64, device="cuda"), max_step=max_step, stream=stream)
                stream.synchronize()
                for _ in range(8000):
                    br.step_device(out, 1e-300, flags, stream=stream)
                stream.synchronize()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append((S, e))

    sizes = [(1800, 1800), (64, 30), (64, 30), (64, 30)]
    threads = [threading.Thread(target=launch, args=(S, m, torch.cuda.Stream())) for S, m in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
