"""Batches of more tubes than the kernels' parameters hold groups of."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tubes(n, cells):
    from electrostatic_b200.negf import CNT
    out = []
    for i in range(n):
        t = CNT(type_id=(17, 0), num_unitcells=cells(i), num_modes=2, contact_mu=(0.0, -0.3),
                contact_T=(300.0, 300.0), eq_integration_pts=(8, 8, 16), noneq_integration_pts=(32,),
                E_zPlus_imag=1e-3)
        U = 0.1 * np.sin(t.site_positions() + i)
        t.set_potential(U, (U[0], U[-1]))
        out.append(t)
    return out


@pytest.fixture
def two_pass():
    """The form by groups for every length."""
    from electrostatic_b200.negf import SCHEDULE_AUTO, SCHEDULE_TWO_PASS, TUNE_SCHEDULE, set_tuning
    set_tuning(TUNE_SCHEDULE, SCHEDULE_TWO_PASS)
    yield
    set_tuning(TUNE_SCHEDULE, SCHEDULE_AUTO)


@pytest.mark.parametrize("n", [33, 65, 100, 200])
def test_batch_equals_single_tubes(two_pass, n):
    """Each tube's charge in the batch is its charge alone (the sums over the
    chains run in another order: rounding), on both sides of one segment."""
    from electrostatic_b200.negf import compute_charge
    tubes = _tubes(n, lambda i: 1 + i % 9)
    Q = compute_charge(tubes)
    off = 0
    for t in tubes:
        q = t.Solve_NEGF()
        assert np.abs(Q[off:off + len(q)] - q).max() <= 1e-12 * np.abs(q).max()
        off += len(q)
    # changed potentials and contacts reach the next call
    for i, t in enumerate(tubes):
        t.set_potential(np.full(t.num_field_sites, 0.01 * i), (0.01 * i, 0.005 * i))
    Q = compute_charge(tubes)
    q = tubes[-1].Solve_NEGF()
    assert np.abs(Q[-len(q):] - q).max() <= 1e-12 * np.abs(q).max()


def test_time_of_many_tubes(two_pass):
    """32 times the tubes of a launch that leaves the GPU nearly empty: far from
    32 times the time (a block that walks the table of groups took 24 times)."""
    import torch
    from electrostatic_b200.negf import ChargePlan

    def time_of(n):
        tubes = _tubes(n, lambda i: 30 + i % 3)
        Q = torch.zeros(sum(t.num_field_sites for t in tubes), dtype=torch.float64, device="cuda")
        plan = ChargePlan(tubes, Q)
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        best = 1e30
        for _ in range(6):
            ev[0].record()
            for _ in range(10):
                plan.launch()
            ev[1].record()
            torch.cuda.synchronize()
            best = min(best, ev[0].elapsed_time(ev[1]))
        plan.close()
        return best
    assert time_of(512) <= 10.0 * time_of(16)
