"""The FP64 ring-block kernels by per-atom potentials.

Without them an FP64 tube's ring-uniform potential runs as the ring's Fourier
modes; here the same potential goes to the blocks: every ring size against the
dense-block oracle, long tubes and decimated leads against the modes, the
benchmark's 600 blocks against both, and the chains' inversion by itself."""
import os

import numpy as np
import pytest

from test_gpu_fullsize import config3  # noqa: F401 - fixture
from test_gpu_realspace import TOL, _bias_kw, _cplx_pack, _eq_kw, _tiles
from test_gpu_parity import _pair, _rel

pytestmark = pytest.mark.gpu


def _atoms(U, m):
    import torch
    return torch.tensor(np.repeat(np.asarray(U), m).reshape(-1, m), device="cuda")


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("m", range(1, 17))
def test_blocks_of_every_ring_size_against_block_oracle(oracle, m, bias):
    """Uniform rings, then atoms of their own; 3 and 4 blocks on the two sides."""
    import torch
    kw = _bias_kw(m, 3 + m % 2) if bias else _eq_kw(m, 3 + m % 2, num_modes=1)
    g, o = _pair(oracle, seed=60 + m, **kw)
    y = g.site_positions()
    U = 0.15 * np.cos(2.0 * y) + 0.1 * (y - y[0]) / (y[-1] - y[0])
    for t in (g, o):
        t.set_potential(U, (U[0], U[-1]))
    assert _rel(g.realspace_charge(U_atoms=_atoms(U, m)), o.rs_charge(nthreads=8)) <= TOL
    Ua = np.repeat(U, m).reshape(-1, m) + 0.05 * np.random.default_rng(m).standard_normal((len(U), m))
    Qg, Qo = g.realspace_charge(U_atoms=torch.tensor(Ua, device="cuda")), o.rs_charge(Uatoms=Ua, nthreads=8)
    assert _rel(Qg, Qo) <= TOL


@pytest.mark.parametrize("extra", [dict(), dict(use_decimation=1)])
@pytest.mark.parametrize("bias", [False, True])
def test_blocks_equal_all_modes(bias, extra):
    """300 blocks of (13,0) (40 with decimated leads): the blocks, the ring's
    modes of the real-space call and the mode-space pass over all 7 modes."""
    from electrostatic_b200.negf import CNT
    from electrostatic_b200.workloads import site_potential
    cells = 20 if extra else 150
    pts = dict(eq_integration_pts=(32, 32, 48), **extra)
    if bias:
        g = CNT(**_bias_kw(13, cells, num_modes=7, noneq_integration_pts=(96,), **pts))
    else:
        g = CNT(**_eq_kw(13, cells, **pts))
    U = site_potential(g.site_positions(), 20261203 + 5)
    g.set_potential(U, (U[0], U[-1]))
    Qb, Qm = g.realspace_charge(U_atoms=_atoms(U, 13)), g.Solve_NEGF()
    assert _rel(Qb, Qm) <= TOL and _rel(g.realspace_charge(), Qm) <= TOL, _rel(Qb, Qm)


def test_config3_blocks_match_block_oracle(config3):  # noqa: F811
    from electrostatic_b200.negf import CNT
    kw, U, Qo = config3
    g = CNT(**dict(kw, precision="fp64"))
    assert g.num_field_sites == 1200  # 600 blocks
    g.set_potential(U, (U[0], U[-1]))
    err = _rel(g.realspace_charge(U_atoms=_atoms(U, 13)), Qo)
    print(f"config 3 FP64 blocks: max rel vs block oracle {err:.3e}")
    assert err <= TOL, err


def test_config3_biased_blocks_match_mode_space_and_oracle(oracle):
    """600 blocks at a 0.3 V drain bias and 1e-4 eV broadening: here the products
    of the real axis are differences of large terms (a product tile taken as
    symmetric moved this charge by 40 times its size, which small tubes did not
    show)."""
    from electrostatic_b200.negf import CNT
    from electrostatic_b200.workloads import SEED_BASE, config3_kwargs, site_potential
    kw = config3_kwargs()
    kw.pop("precision")
    kb = dict(kw, contact_mu=(-0.8, -1.1), noneq_integration_pts=(3072,), E_zPlus_imag=1e-4)
    g = CNT(**kb)
    o = oracle.OracleTube(**dict(kb, noneq_percent_intercuts=None))
    U = site_potential(g.site_positions(), SEED_BASE + 3)
    for t in (g, o):
        t.set_potential(U, (U[0], U[-1]))
    Qb = g.realspace_charge(U_atoms=_atoms(U, 13))
    err_m = _rel(Qb, g.Solve_NEGF())
    err_o = _rel(Qb, o.charge(nthreads=max(1, len(os.sched_getaffinity(0)))))
    print(f"config 3 biased blocks: vs mode space {err_m:.3e}, vs oracle {err_o:.3e}")
    assert err_m <= TOL and err_o <= TOL, (err_m, err_o)


@pytest.mark.parametrize("m", range(1, 17))
def test_symmetric_inversion(negf_lib, m):
    """The chains' inversion (sweeps on 2 x 2 blocks, partial pivoting behind a
    large multiplier) on complex symmetric matrices: like E - H - Sigma; with
    leading 2 x 2 blocks singular but for 1e-3 to 1e-14; with a zero diagonal.
    Multipliers of up to 256 in each of 8 blocks at most: residual within 256
    roundings of the condition number."""
    rng = np.random.default_rng(m)
    n = 24
    A = rng.standard_normal((n, m, m)) + 1j * rng.standard_normal((n, m, m))
    A = 0.3 * (A + np.transpose(A, (0, 2, 1)))
    A += np.eye(m)[None] * (2.0 + 0.5j)
    sets = [A]
    if m >= 2:
        B = A.copy()
        for i in range(n):
            B[i, 0, 0] = B[i, 0, 1] ** 2 / B[i, 1, 1] + 10.0 ** -(3 + i % 12)
        Z = A.copy()
        Z[:, np.arange(m), np.arange(m)] = 0.0
        sets += [B, Z]
    for M in sets:
        keep = [i for i in range(len(M)) if np.linalg.cond(M[i]) < 1e10]
        M = M[keep]
        if not len(M):
            continue
        X = _tiles(negf_lib, 6, m, _cplx_pack(M), len(M), 2 * m * m)
        for Mi, Xi in zip(M, X):
            res = np.abs(Mi @ Xi - np.eye(m)).max()
            assert res <= 256 * 16 * 2.3e-16 * max(1.0, np.linalg.cond(Mi)), (res, np.linalg.cond(Mi))
