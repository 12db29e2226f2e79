"""Standing waves between contacts at another potential than the channel.

In a flat channel the modulus of a sweep's state goes up and down with the
wave; at energies where one segment turns it by a quarter period the growth
of one segment and the decay of the next alternate over the whole tube.  The
scaling at the segment boundaries must keep the state in range there (a
scaling by 1 / |q|^2 lets it grow geometrically, to a NaN charge).  Bound: the
repository's FP64 parity bound against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-8


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def _flat(n, u):
    U = np.full(n, u)
    U[0] = U[-1] = 0.0
    return U


@pytest.fixture
def tuning():
    from electrostatic_b200.negf import TUNE_PASS1_PIECES, TUNE_SCHEDULE, set_tuning
    yield set_tuning
    set_tuning(TUNE_PASS1_PIECES, 0)
    set_tuning(TUNE_SCHEDULE, 0)


# 4000 sites: the step of -0.6 eV loses every site of whole sweeps, +0.8 eV those of one direction
CASES = [(1000, -0.6), (1000, 0.8), (2000, -1.0)]


def _tube_and_oracle(oracle, cells, u):
    from electrostatic_b200.negf import CNT
    kw = dict(type_id=(17, 0), num_unitcells=cells, num_modes=2, contact_mu=(0.0, -0.3), contact_T=(300.0, 300.0),
              eq_integration_pts=(16, 16, 32), noneq_integration_pts=(3072,), E_zPlus_imag=1e-5)
    g, o = CNT(**kw), oracle.OracleTube(**kw)
    U = _flat(g.num_field_sites, u)
    for t in (g, o):
        t.set_potential(U, (0.0, 0.0))
    return g, o.charge(nthreads=8)


@pytest.mark.parametrize("cells,u", CASES)
def test_flat_channel_sweeps(oracle, tuning, cells, u):
    from electrostatic_b200.negf import TUNE_PASS1_PIECES
    g, Qo = _tube_and_oracle(oracle, cells, u)
    for P in (0, 1):  # the automatic form, whole sweeps
        tuning(TUNE_PASS1_PIECES, P)
        Qg = g.Solve_NEGF()
        assert np.all(np.isfinite(Qg)) and _rel(Qg, Qo) <= FP64_TOL, (P, _rel(Qg, Qo))


MIXED_TOL = 1e-5


@pytest.mark.parametrize("cells,u", CASES)
def test_flat_channel_fused(oracle, tuning, cells, u):
    from electrostatic_b200.negf import SCHEDULE_FUSED, TUNE_SCHEDULE
    g, Qo = _tube_and_oracle(oracle, cells, u)
    tuning(TUNE_SCHEDULE, SCHEDULE_FUSED)
    Qg = g.Solve_NEGF()
    assert np.all(np.isfinite(Qg)) and _rel(Qg, Qo) <= FP64_TOL, _rel(Qg, Qo)


@pytest.mark.parametrize("cells,u", CASES)
def test_flat_channel_fp64_chains_of_a_mixed_tube(oracle, tuning, cells, u):
    """Mostly FP32 work: the FP64 chains near the axis ride along, in both schedules."""
    from electrostatic_b200.negf import CNT, SCHEDULE_FUSED, SCHEDULE_TWO_PASS, TUNE_SCHEDULE
    kw = dict(type_id=(17, 0), num_unitcells=cells, num_modes=2, contact_mu=(0.0, -0.3), contact_T=(300.0, 300.0),
              eq_integration_pts=(900, 900, 1500), noneq_integration_pts=(3072,), E_zPlus_imag=1e-5)
    o = oracle.OracleTube(**kw)
    g = CNT(**kw, precision="mixed")
    U = _flat(g.num_field_sites, u)
    for t in (g, o):
        t.set_potential(U, (0.0, 0.0))
    Qo = o.charge(nthreads=8)
    for schedule in (SCHEDULE_FUSED, SCHEDULE_TWO_PASS):
        tuning(TUNE_SCHEDULE, schedule)
        Qg = g.Solve_NEGF()
        assert np.all(np.isfinite(Qg)) and _rel(Qg, Qo) <= MIXED_TOL, (schedule, _rel(Qg, Qo))
