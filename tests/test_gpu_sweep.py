"""FP64 passes by boundary states and segments (csrc/negf_sweep.cu) against the
oracle, at the sizes where their tiling can go wrong: tubes shorter than one
16-site segment (2-site segments), one segment, the overlapping last segment
(N not a multiple of 16), more than 8 and more than 32 segments, chain counts
that are no multiple of 32 or of the chains of a unit; both ways to the
boundary states (sweeps, and the scan over segments, with more segments than
threads).  Bound: the repository's FP64 parity bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-8
SWEEP, SCAN = 1, 2  # pieces setting: one sweep per chain, parallel in length


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


@pytest.fixture
def pieces():
    from electrostatic_b200.negf import TUNE_PASS1_PIECES, set_tuning
    yield lambda v: set_tuning(TUNE_PASS1_PIECES, v)
    set_tuning(TUNE_PASS1_PIECES, 0)


# (type_id, unit cells): N = 4 * cells for zigzag, 2 * cells for the chiral (13, 2)
LENGTHS = [((13, 2), 1), ((13, 2), 3), ((17, 0), 2), ((13, 2), 7), ((17, 0), 4), ((13, 2), 9), ((13, 2), 15),
           ((17, 0), 8), ((17, 0), 9), ((17, 0), 32), ((13, 2), 65), ((17, 0), 129), ((17, 0), 130)]


@pytest.mark.parametrize("way", [SWEEP, SCAN])
@pytest.mark.parametrize("tid,cells", LENGTHS)
def test_segments_match_oracle(oracle, pieces, way, tid, cells):
    from electrostatic_b200.negf import CNT
    from electrostatic_b200.workloads import site_potential
    # 3 modes and 9 + 9 + 15 contour, 11 + 20 + 10 real-axis points: 99 and 123 chains
    kw = dict(type_id=tid, num_unitcells=cells, num_modes=3, contact_mu=(0.05, -0.25), contact_T=(300.0, 320.0),
              eq_integration_pts=(9, 9, 15), noneq_integration_pts=(11, 20, 10), E_zPlus_imag=1e-3)
    pieces(way)
    g = CNT(**kw)
    U = site_potential(g.site_positions(), 500 + cells, amp=0.3, ramp=0.2)
    g.set_potential(U, (U[0], U[-1]))
    o = oracle.OracleTube(**kw)
    o.set_potential(U, (U[0], U[-1]))
    Qg, Qo = g.Solve_NEGF(), o.charge(nthreads=8)
    assert _rel(Qg, Qo) <= FP64_TOL, (g.num_field_sites, _rel(Qg, Qo))
    assert np.array_equal(g.Solve_NEGF(), Qg)  # fixed order of every sum


@pytest.mark.parametrize("way", [SWEEP, SCAN])
def test_vanishing_hopping_and_decimated_leads(oracle, pieces, way):
    """A mode whose beta is zero to rounding ((10,0), J = 5: the dimers decouple
    and lambda vanishes), and the reference's decimation in the leads."""
    from electrostatic_b200.negf import CNT
    pieces(way)
    for extra in (dict(), dict(use_decimation=1)):
        kw = dict(type_id=(10, 0), num_unitcells=11, num_modes=6, contact_mu=(0.0, -0.3), contact_T=(300.0, 300.0),
                  eq_integration_pts=(8, 8, 12), noneq_integration_pts=(24,), E_zPlus_imag=1e-3, **extra)
        g = CNT(**kw)
        assert np.min(np.abs(g.modes()[2])) < 1e-12
        y = g.site_positions()
        U = 0.1 * np.cos(y) + 0.05 * (y - y[0]) / (y[-1] - y[0])
        g.set_potential(U, (U[0], U[-1]))
        o = oracle.OracleTube(**kw)
        o.set_potential(U, (U[0], U[-1]))
        Qg, Qo = g.Solve_NEGF(), o.charge(nthreads=8)
        assert _rel(Qg, Qo) <= FP64_TOL, (extra, _rel(Qg, Qo))


@pytest.mark.parametrize("way", [SWEEP, SCAN])
def test_more_segments_than_threads(pieces, way):
    """9000 sites (563 segments, 512 threads of a scan block) and 40 chains: the
    two ways and a batch with a short tube agree to the rounding of their sums."""
    from electrostatic_b200.negf import CNT, compute_charge
    from electrostatic_b200.workloads import site_potential

    def tube(cells, seed):
        t = CNT(type_id=(17, 0), num_unitcells=cells, num_modes=2, contact_mu=(0.0, -0.2), contact_T=(300.0, 300.0),
                eq_integration_pts=(4, 4, 6), noneq_integration_pts=(6,), E_zPlus_imag=1e-3)
        U = site_potential(t.site_positions(), seed, amp=0.2, ramp=0.2)
        t.set_potential(U, (U[0], U[-1]))
        return t
    long_, short = tube(2250, 3), tube(2, 4)
    pieces(SWEEP)
    ref = [long_.Solve_NEGF(), short.Solve_NEGF()]
    pieces(way)
    # 1e-11: the transfer matrices accumulate one rounding per site (9000 eps = 2e-12) where the sweep renormalises
    assert _rel(long_.Solve_NEGF(), ref[0]) <= 1e-11
    both = compute_charge([short, long_])
    assert _rel(both, np.concatenate([ref[1], ref[0]])) <= 1e-11


def test_many_tubes_read_their_groups_from_memory(oracle):
    """40 tubes (80 groups: more than stand in the kernels' parameters), lengths on both sides of one segment."""
    from electrostatic_b200.negf import CNT, compute_charge
    tubes, refs = [], []
    for i in range(40):
        kw = dict(type_id=(17, 0), num_unitcells=1 + i % 7, num_modes=1 + i % 3, contact_mu=(0.0, -0.1 - 0.005 * i),
                  contact_T=(300.0, 300.0), eq_integration_pts=(4, 4, 6), noneq_integration_pts=(7,), E_zPlus_imag=1e-3)
        t = CNT(**kw)
        U = 0.1 * np.sin(t.site_positions() + i)
        t.set_potential(U, (U[0], U[-1]))
        o = oracle.OracleTube(**kw)
        o.set_potential(U, (U[0], U[-1]))
        tubes.append(t)
        refs.append(o.charge(nthreads=4))
    Q = compute_charge(tubes)
    off = 0
    for r in refs:
        assert _rel(Q[off:off + len(r)], r) <= FP64_TOL
        off += len(r)


# N = 4, 6 (2-site segments), 16, 18, 34 and 516 (33 segments: two blocks of them); on two sites the
# oracle counts the drain site, which is also N/2, twice
@pytest.mark.parametrize("tid,cells", [((17, 0), 1), ((13, 2), 3), ((17, 0), 4), ((13, 2), 9), ((13, 2), 17), ((17, 0), 129)])
def test_transport_segments_match_oracle(oracle, tid, cells):
    """Density of states, transmission, LDOS, current and its probes at the edges of the segment tiling."""
    from electrostatic_b200.negf import CNT
    from electrostatic_b200.workloads import site_potential
    kw = dict(type_id=tid, num_unitcells=cells, num_modes=3, contact_mu=(0.0, -0.3), contact_T=(300.0, 300.0),
              noneq_integration_pts=(17, 24), noneq_percent_intercuts=(40.0,), E_zPlus_imag=1e-4)
    g, o = CNT(**kw), oracle.OracleTube(**kw)
    U = site_potential(g.site_positions(), 900 + cells, amp=0.2, ramp=0.2)
    for t in (g, o):
        t.set_potential(U, (U[0], U[-1]))
    d, od = g.Compute_DensityOfStates(ldos=True), o.dos(faithful=True, nthreads=8, ldos=True)
    for key in ("dos", "T", "conductance", "ldos"):
        assert _rel(d[key], od[key]) <= FP64_TOL, (key, _rel(d[key], od[key]))
    I, probes, _ = g.Compute_Current(integrand=True)
    oI, oprobes = o.current(nthreads=8, probes=True)
    assert _rel(I, oI) <= FP64_TOL and _rel(probes, oprobes) <= FP64_TOL


@pytest.mark.parametrize("cells", [4000, 4001, 4036, 5125])
def test_sweeps_in_pieces(pieces, cells):
    """Long tubes of a middling number of chains: sweeps in pieces (chosen by the
    estimate) against whole ones, with a last piece of one segment more, whole and
    overlapping last segments, the mode of a vanishing hopping and a short tube in
    the same launch.  1e-11: one rounding per site of the matrices (2e4 eps = 5e-12)."""
    import torch
    from electrostatic_b200.negf import CNT, ChargePlan
    from electrostatic_b200.workloads import site_potential

    def tube(type_id, n, modes, seed):
        t = CNT(type_id=type_id, num_unitcells=n, num_modes=modes, contact_mu=(0.0, -0.2), contact_T=(300.0, 300.0),
                eq_integration_pts=(16, 16, 32), noneq_integration_pts=(70,), E_zPlus_imag=1e-3)
        U = site_potential(t.site_positions(), seed, amp=0.2, ramp=0.2)
        t.set_potential(U, (U[0], U[-1]))
        return t
    tubes = [tube((16, 0), cells, 8, 3), tube((17, 0), 40, 2, 4), tube((17, 0), 3, 2, 5)]
    pieces(SWEEP)
    ref = [t.Solve_NEGF() for t in tubes]
    pieces(0)
    assert _rel(tubes[0].Solve_NEGF(), ref[0]) <= 1e-11
    Q = torch.zeros(sum(len(r) for r in ref), dtype=torch.float64, device="cuda")
    plan = ChargePlan(tubes, Q)
    assert 1 < plan.info()["pieces"] < 200
    plan.launch()
    torch.cuda.synchronize()
    assert _rel(Q.cpu().numpy(), np.concatenate(ref)) <= 1e-11
