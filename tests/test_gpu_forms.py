"""The form of a batch's FP64 chains (groups or the fused schedule): the
automatic choice and the autotuner's against both of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tubes(sites, energies, modes=8, **extra):
    from electrostatic_b200.negf import CNT
    from electrostatic_b200.workloads import site_potential
    out = []
    for i, n in enumerate(sites):
        E = energies[i % len(energies)]
        t = CNT(type_id=(17, 0), num_unitcells=n // 4, num_modes=modes, contact_mu=(0.0, -0.3),
                contact_T=(300.0, 300.0), eq_integration_pts=(E // 8, E // 8, E // 4),
                noneq_integration_pts=(E // 2,), E_zPlus_imag=1e-3, **extra)
        U = site_potential(t.site_positions(), i, amp=0.2, ramp=0.2)
        t.set_potential(U, (U[0], U[-1]))
        out.append(t)
    return out


@pytest.fixture
def schedule():
    from electrostatic_b200.negf import TUNE_SCHEDULE, set_tuning
    yield lambda v: set_tuning(TUNE_SCHEDULE, v)
    set_tuning(TUNE_SCHEDULE, 0)


@pytest.mark.parametrize("sites", [[4], [8], [28], [16, 8, 12], [64] * 4, [48, 8, 8, 64], [128], [300, 8, 1200]])
def test_forms_agree(schedule, sites):
    """Automatic, groups and fused give one charge (calls and plans); 1e-11: the orders of the sums and one
    rounding per site of the matrices."""
    import torch
    from electrostatic_b200.negf import SCHEDULE_FUSED, SCHEDULE_TWO_PASS, ChargePlan, compute_charge, last_stats
    tubes = _tubes(sites, [96, 160])
    out = {}
    for s in (0, SCHEDULE_TWO_PASS, SCHEDULE_FUSED):
        schedule(s)
        out[s] = compute_charge(tubes)
        st = last_stats()
        if s:
            assert st["schedule"] == s
        elif max(sites) < 32:
            assert st["schedule"] == SCHEDULE_FUSED and st["pieces"] == 1
        for tune in (False, True):
            Q = torch.zeros(sum(sites), dtype=torch.float64, device="cuda")
            plan = ChargePlan(tubes, Q, autotune=tune)
            plan.launch()
            torch.cuda.synchronize()
            q = Q.cpu().numpy()
            assert np.abs(q - out[s]).max() <= 1e-11 * np.abs(q).max(), (s, tune)
            plan.close()
    for s in (SCHEDULE_TWO_PASS, SCHEDULE_FUSED):
        assert np.abs(out[s] - out[0]).max() <= 1e-11 * np.abs(out[0]).max(), s


def _time(plan):
    import torch
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    best = 1e30
    for _ in range(8):
        ev[0].record()
        for _ in range(10):
            plan.launch()
        ev[1].record()
        torch.cuda.synchronize()
        best = min(best, ev[0].elapsed_time(ev[1]))
    return best


@pytest.mark.parametrize("sites,energies", [([8] * 16, [8000]), ([64, 48, 8, 8], [36, 60, 280, 390]),
                                            ([1200], [500])])
def test_the_faster_form_runs(schedule, sites, energies):
    """Well inside each form's range (the other one takes 1.5 times as long or more)."""
    import torch
    from electrostatic_b200.negf import SCHEDULE_FUSED, SCHEDULE_TWO_PASS, ChargePlan
    tubes = _tubes(sites, energies)
    Q = torch.zeros(sum(sites), dtype=torch.float64, device="cuda")
    times = {}
    for s in (SCHEDULE_TWO_PASS, SCHEDULE_FUSED, 0):
        schedule(s)
        plan = ChargePlan(tubes, Q)
        times[s] = _time(plan)
        plan.close()
    tuned = ChargePlan(tubes, Q, autotune=True)
    t = _time(tuned)
    tuned.close()
    best = min(times[SCHEDULE_TWO_PASS], times[SCHEDULE_FUSED])
    assert times[0] <= 1.2 * best and t <= 1.2 * best, (times, t)
