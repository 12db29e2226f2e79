"""Host results are ordinary numpy memory."""
import gc
import subprocess
import sys

import numpy as np
import pytest


def test_result_memory_needs_no_torch():
    code = ("import sys; sys.modules['torch'] = None\n"
            "from electrostatic_b200.negf import _ResultPool\n"
            "p = _ResultPool(); a = p.array(20000); where = a.ctypes.data; a[:] = 1.0; del a\n"
            "assert p.array(20000).ctypes.data == where and p._bytes == 1 << 18\n")
    subprocess.run([sys.executable, "-c", code], check=True, timeout=120)


def test_views_keep_a_block_in_use():
    from electrostatic_b200.negf import _ResultPool
    pool = _ResultPool()
    a = pool.array(20000)
    view = a.reshape(100, 200)[3:, ::2]
    view[:] = 7.0
    where = a.ctypes.data
    del a
    gc.collect()
    b = pool.array(20000)
    b[:] = 1.0
    assert b.ctypes.data != where and np.all(view == 7.0)
    keep = [pool.array(1 << 20) for _ in range(12)]  # past the bound: arrays of their own
    assert pool._bytes <= pool.LIMIT and len({k.ctypes.data for k in keep}) == 12
    del keep, b, view
    gc.collect()
    pool.clear()
    assert pool._bytes == 0


@pytest.mark.gpu
def test_results_are_pageable_and_owned():
    """A charge owns its memory (it can be resized); neither it nor a local density
    of states is page-locked, so an upload that the caller enqueues has read it when
    the enqueuing call returns."""
    import torch
    from electrostatic_b200.negf import CNT
    t = CNT(type_id=(17, 0), num_unitcells=8000, num_modes=1, contact_mu=(0.0, -0.2), contact_T=(300.0, 300.0),
            eq_integration_pts=(4, 4, 6), noneq_integration_pts=(6,), E_zPlus_imag=1e-3, flatband_dos_integration_pts=6)
    t.set_potential(np.zeros(t.num_field_sites), (0.0, 0.0))
    Q, ldos = t.Solve_NEGF(), t.Compute_DensityOfStates(ldos=True)["ldos"]
    for x in (Q, ldos):
        assert x.nbytes > 1 << 16 and not torch.from_numpy(x).is_pinned()
    keep = Q.copy()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)  # the copy below runs after this
        up = torch.from_numpy(Q).to("cuda", non_blocking=True)
    Q[:] = -1.0
    torch.cuda.synchronize()
    assert np.array_equal(up.cpu().numpy(), keep)
    Q.resize(10, refcheck=False)
