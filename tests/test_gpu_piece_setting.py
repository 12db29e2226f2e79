"""NEGF_TUNE_PASS1_PIECES for FP64 chains: P pieces of each tube, and the scan
over segments where pieces of 128 sites are too long for the setting."""
import numpy as np
import pytest

from test_gpu_sweep import FP64_TOL, LENGTHS, _rel

pytestmark = pytest.mark.gpu

SCAN = 1024  # pieces shorter than 128 sites for every tube below


@pytest.fixture
def pieces():
    from electrostatic_b200.negf import TUNE_PASS1_PIECES, set_tuning
    yield lambda v: set_tuning(TUNE_PASS1_PIECES, v)
    set_tuning(TUNE_PASS1_PIECES, 0)


def _tube(cells, modes, eq, ne, seed=3, tid=(17, 0)):
    from electrostatic_b200.negf import CNT
    from electrostatic_b200.workloads import site_potential
    t = CNT(type_id=tid, num_unitcells=cells, num_modes=modes, contact_mu=(0.0, -0.2), contact_T=(300.0, 300.0),
            eq_integration_pts=eq, noneq_integration_pts=(ne,), E_zPlus_imag=1e-3)
    U = site_potential(t.site_positions(), seed, amp=0.2, ramp=0.2)
    t.set_potential(U, (U[0], U[-1]))
    return t


# 256 sites: two pieces of the minimal length; 260: the last 4 sites join the piece before; 4000: up to 32 pieces
@pytest.mark.parametrize("cells", [33, 64, 65, 97, 1000])
@pytest.mark.parametrize("P", [2, 3, 8, 64])
def test_pieces_of_the_setting(pieces, cells, P):
    """Sweeps in pieces (four launches) for tubes of more than 128 sites where the
    setting leaves pieces of at least 128 sites; the charge of whole sweeps.
    1e-11: one rounding per site of the matrices."""
    from electrostatic_b200.negf import last_stats
    t = _tube(cells, 2, (16, 16, 32), 40)
    pieces(1)
    ref = t.Solve_NEGF()
    pieces(P)
    Q, st = t.Solve_NEGF(), last_stats()
    assert _rel(Q, ref) <= 1e-11
    assert st["pieces"] == P
    N = t.num_field_sites
    L = -(-N // (128 * P)) * 128  # sites of a piece; a last piece of one segment joins the one before
    n = -(-N // L) - (1 if 0 < N % L <= 16 else 0)
    assert st["kernel_launches"] == (4 if N >= 128 * P and n > 1 else 3)


def test_many_chains_keep_pieces(pieces):
    """P = 64 on 4000 sites: shorter than 128 sites, but the scan of 30 000 chains is the slower form."""
    from electrostatic_b200.negf import last_stats
    t = _tube(1000, 8, (256, 256, 512), 2600)
    pieces(1)
    ref = t.Solve_NEGF()
    pieces(64)
    assert _rel(t.Solve_NEGF(), ref) <= 1e-11
    assert last_stats()["kernel_launches"] == 4


def test_batch_of_long_and_short_tubes_in_pieces(pieces):
    """Each tube in its own P pieces; tubes of up to 128 sites and of fewer than 16 in one."""
    from electrostatic_b200.negf import compute_charge
    tubes = [_tube(n, 2, (16, 16, 32), 40, seed=n) for n in (1000, 300, 20, 3)]
    pieces(1)
    ref = [t.Solve_NEGF() for t in tubes]
    for P in (2, 8):
        pieces(P)
        assert _rel(compute_charge(tubes), np.concatenate(ref)) <= 1e-11


@pytest.mark.parametrize("tid,cells", LENGTHS)
def test_scan_matches_oracle(oracle, pieces, tid, cells):
    from electrostatic_b200.negf import CNT, last_stats
    from electrostatic_b200.workloads import site_potential
    kw = dict(type_id=tid, num_unitcells=cells, num_modes=3, contact_mu=(0.05, -0.25), contact_T=(300.0, 320.0),
              eq_integration_pts=(9, 9, 15), noneq_integration_pts=(11, 20, 10), E_zPlus_imag=1e-3)
    pieces(SCAN)
    g, o = CNT(**kw), oracle.OracleTube(**kw)
    U = site_potential(g.site_positions(), 500 + cells, amp=0.3, ramp=0.2)
    for t in (g, o):
        t.set_potential(U, (U[0], U[-1]))
    Qg, Qo = g.Solve_NEGF(), o.charge(nthreads=8)
    assert _rel(Qg, Qo) <= FP64_TOL, _rel(Qg, Qo)
    assert last_stats()["kernel_launches"] == 3


def test_scan_of_more_segments_than_threads(pieces):
    """9000 sites (563 segments, 512 threads of a scan block)."""
    from electrostatic_b200.negf import last_stats
    t = _tube(2250, 2, (4, 4, 6), 6)
    pieces(1)
    ref = t.Solve_NEGF()
    pieces(SCAN)
    assert _rel(t.Solve_NEGF(), ref) <= 1e-11
    assert last_stats()["kernel_launches"] == 3
