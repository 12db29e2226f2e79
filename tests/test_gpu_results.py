"""Page-locked memory of large host results: lifetime and bound."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_result_pool_lifetime_and_bound():
    from electrostatic_b200.negf import _ResultPool
    pool = _ResultPool()
    assert pool.array(100).base is None  # small: an ordinary array
    a = pool.array(20000)
    assert a.dtype == np.float64 and a.shape == (20000,) and a.flags.writeable
    where, view = a.ctypes.data, a.reshape(100, 200)[3:, ::2]
    view[:] = 7.0
    del a
    gc.collect()
    b = pool.array(20000)  # the view still holds the first block
    assert b.ctypes.data != where
    b[:] = 1.0
    assert np.all(view == 7.0)
    del view
    gc.collect()
    assert pool.array(16385).ctypes.data == where  # the same power of two
    keep = [pool.array(1000000) for _ in range(12)]
    assert len({k.ctypes.data for k in keep}) == 12 and pool._bytes <= pool.LIMIT
    del keep, b
    gc.collect()
    pool.clear()
    assert pool._bytes == 0


def test_results_of_calls_are_independent():
    """Charges and densities of states of two calls do not share memory."""
    from electrostatic_b200.negf import CNT
    from electrostatic_b200.workloads import site_potential
    t = CNT(type_id=(17, 0), num_unitcells=3000, num_modes=1, contact_mu=(0.0, -0.2), contact_T=(300.0, 300.0),
            eq_integration_pts=(4, 4, 6), noneq_integration_pts=(6,), E_zPlus_imag=1e-3)
    out = []
    for seed in (3, 4):
        U = site_potential(t.site_positions(), seed, amp=0.2, ramp=0.2)
        out.append((t.Solve_NEGF(U, (U[0], U[-1])), t.Compute_DensityOfStates(ldos=True)["ldos"]))
    first = [x.copy() for x in out[0]]
    U = site_potential(t.site_positions(), 3, amp=0.2, ramp=0.2)
    again = (t.Solve_NEGF(U, (U[0], U[-1])), t.Compute_DensityOfStates(ldos=True)["ldos"])
    for a, b, c in zip(first, out[0], again):
        assert np.array_equal(a, b) and np.array_equal(a, c)
    assert not np.array_equal(out[0][0], out[1][0])
