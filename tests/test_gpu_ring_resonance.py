"""Real-axis energies that pass the potential of whole rings.

The two halves of a real-axis chain meet at surface functions that are as large
as 1 / Im E in some of the ring's modes there; the columns of G across the
meeting point are formed without their differences.  Potential: one grid
energy on every atom, on the rings a or b, on the two rings that meet, and on
random atoms.  Bound: the repository's FP64 parity bound against the dense-block
oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-8


@pytest.mark.parametrize("eta", [1e-4, 1e-6, 1e-8])
@pytest.mark.parametrize("m,cells", [(4, 2), (4, 5), (5, 5), (7, 5), (10, 3), (13, 2), (13, 3), (13, 4), (13, 5)])
def test_grid_energy_on_ring_potentials(oracle, m, cells, eta):
    import torch
    from electrostatic_b200.negf import CNT
    kw = dict(type_id=(m, 0), num_unitcells=cells, num_modes=1, contact_mu=(0.0, -0.3), contact_T=(300.0, 320.0),
              eq_integration_pts=(16, 16, 24), noneq_integration_pts=(48,), E_pole_max=3.0, E_zPlus_imag=eta)
    g = CNT(**kw)
    o = oracle.OracleTube(**kw, noneq_percent_intercuts=None)
    n = g.num_field_sites
    for t in (g, o):
        t.set_potential(np.zeros(n), (0.0, 0.0))
    e = g.energy_points(3)[0][20].real
    rng = np.random.default_rng(m)
    base = 0.05 * rng.standard_normal((n, m))
    for where in ("all", "a", "b", "middle", "some"):
        Ua = base.copy()
        if where == "all":
            Ua[:] = e
        elif where in "ab":
            Ua["ab".index(where)::2] = e
        elif where == "middle":
            Ua[n // 2 - 1:n // 2 + 1] = e
        else:
            Ua[rng.random((n, m)) < 0.5] = e
        Qg = g.realspace_charge(U_atoms=torch.tensor(Ua, device="cuda"))
        Qo = o.rs_charge(Uatoms=Ua, nthreads=8)
        err = float(np.abs(Qg - Qo).max() / np.abs(Qo).max())
        assert err <= TOL, (where, err)
