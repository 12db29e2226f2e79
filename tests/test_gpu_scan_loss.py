"""The scan over segments where its products lose digits.

Periodic and random potentials at a small broadening: at some energies the wave
decays through a stop band or meets a resonance, and a product of transfer
matrices, or of one with a state, is a small difference of large terms.  Such a
chain is swept.  Against the oracle at the repository's FP64 parity bound, and
against whole sweeps at 1e-9: one product in 2^8 keeps 1e-13 of a state and the
resonance's weight in the charge is below 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-8


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


def _cos(n, period):
    return 0.5 * np.cos(2.0 * np.pi * np.arange(n) / period)


CASES = {
    "stop_band_12": (dict(type_id=(12, 0), num_unitcells=98, num_modes=2, gamma=1.0, contact_mu=(0.0, -0.2),
                          contact_T=(77.0, 300.0), noneq_integration_pts=(300,), E_zPlus_imag=2.321353500763346e-06),
                     lambda n: _cos(n, 32.5)),
    "stop_band_13": (dict(type_id=(13, 0), num_unitcells=201, num_modes=5, gamma=1.0, contact_mu=(0.0, -0.5),
                          contact_T=(400.0, 300.0), noneq_integration_pts=(64,), E_zPlus_imag=7.293506643390702e-07),
                     lambda n: _cos(n, 32)),
    "stop_band_10": (dict(type_id=(10, 0), num_unitcells=638, num_modes=5, gamma=2.7, contact_mu=(0.0, -0.5),
                          contact_T=(77.0, 300.0), noneq_integration_pts=(64,), E_zPlus_imag=3.05932851333104e-06),
                     lambda n: _cos(n, 32)),
    "random": (dict(type_id=(17, 0), num_unitcells=262, num_modes=5, gamma=1.0, contact_mu=(0.0, -1.0),
                    contact_T=(400.0, 300.0), noneq_integration_pts=(257,), E_zPlus_imag=1.3e-06),
               lambda n: np.random.default_rng(20).normal(0.0, 0.5, n)),
    "short_segments": (dict(type_id=(12, 0), num_unitcells=3, num_modes=2, gamma=1.0, contact_mu=(0.0, -0.2),
                            contact_T=(77.0, 300.0), noneq_integration_pts=(300,), E_zPlus_imag=1e-7),
                       lambda n: _cos(n, 5)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_scan_keeps_its_digits(oracle, name):
    from electrostatic_b200.negf import (CNT, SCHEDULE_AUTO, SCHEDULE_TWO_PASS, TUNE_PASS1_PIECES, TUNE_SCHEDULE,
                                         set_tuning)
    kw, make = CASES[name]
    kw = dict(kw, eq_integration_pts=(8, 8, 16))
    g, o = CNT(**kw), oracle.OracleTube(**kw)
    U = make(g.num_field_sites)
    for t in (g, o):
        t.set_potential(U, (U[0], U[-1]))
    Qo = o.charge(nthreads=8)
    set_tuning(TUNE_SCHEDULE, SCHEDULE_TWO_PASS)
    try:
        set_tuning(TUNE_PASS1_PIECES, 1)
        whole = g.Solve_NEGF()
        set_tuning(TUNE_PASS1_PIECES, 1024)
        scan = g.Solve_NEGF()
    finally:
        set_tuning(TUNE_PASS1_PIECES, 0)
        set_tuning(TUNE_SCHEDULE, SCHEDULE_AUTO)
    assert _rel(scan, Qo) <= FP64_TOL, _rel(scan, Qo)
    assert _rel(scan, whole) <= 1e-9, _rel(scan, whole)
    assert _rel(g.Solve_NEGF(), Qo) <= FP64_TOL
