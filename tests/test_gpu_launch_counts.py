"""negf_stats.kernel_launches against the launches of each form of a charge call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(cells, **kw):
    from electrostatic_b200.negf import CNT, last_stats
    d = dict(type_id=(17, 0), num_unitcells=cells, num_modes=2, contact_mu=(0.0, -0.2), contact_T=(300.0, 300.0),
             eq_integration_pts=(16, 16, 32), noneq_integration_pts=(70,), E_zPlus_imag=1e-3)
    t = CNT(**dict(d, **kw))
    t.set_potential(np.zeros(t.num_field_sites), (0.0, 0.0))
    t.Solve_NEGF()
    return last_stats()


@pytest.fixture
def two_pass():
    from electrostatic_b200.negf import SCHEDULE_AUTO, SCHEDULE_TWO_PASS, TUNE_SCHEDULE, set_tuning
    set_tuning(TUNE_SCHEDULE, SCHEDULE_TWO_PASS)
    yield
    set_tuning(TUNE_SCHEDULE, SCHEDULE_AUTO)


def test_kernel_launches_of_each_form(two_pass):
    assert _call(3)["kernel_launches"] == 3      # 12 sites, 2-site segments: states, segments, reduction
    assert _call(100)["kernel_launches"] == 3    # the scan over segments, segments, reduction
    st = _call(4000, type_id=(16, 0), num_modes=8)
    assert st["pieces"] > 1 and st["pieces"] < 200  # sweeps in pieces
    assert st["kernel_launches"] == 4            # and their matrices before
