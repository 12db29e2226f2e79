"""Timed cases of the NEGF charge engine: what its users have it compute.

Every case goes through the package's public entry points (CNT, compute_charge,
ChargePlan, BatchSCF, realspace_charge, the transport characteristics, the
surrogate operator).  A case is a dict of plain values; its "kind" names the
entry point:

  solve      CNT.Solve_NEGF with the potential and the charge on the host: the
             call that a transport loop makes once per iteration and tube
  charge     set_potential_device + compute_charge into a device buffer: the
             same pass inside a program that keeps its vectors on the GPU
  batch      ChargePlan.launch over an uneven set of tubes (one launch per
             iteration of a multi-tube device)
  scf        BatchSCF.solve: one gate point of a batch (potential update, charge
             plan and Broyden step, replayed as a CUDA graph)
  rs         CNT.realspace_charge: ring-block Green's function, with per-atom
             potentials (disorder, charged defects) or a ring-uniform one
  transport  Compute_DensityOfStates with the LDOS, and Compute_Current: the
             post-processing of a bias point
  train      one gradient of the surrogate operator (forward, loss, backward)

All inputs are drawn from the seed.  `exact` evaluates the same charge,
density of states and current in plain complex128 torch: quadrature points from the
published formulas, scalar recursions per mode, ring-by-ring matrix recursions for
per-atom potentials.
"""
from __future__ import annotations

import math

import numpy as np
import torch

KB_EV = 8.617333262e-5       # Boltzmann constant [eV/K]
Q_E = 1.602176634e-19        # elementary charge [C]
H_EV = 4.135667696e-15       # Planck constant [eV s]
ACC = 1.42e-10               # carbon-carbon distance [m]
GAMMA = 2.5                  # hopping [eV]
TAIL = 14.0                  # Fermi tail of the energy limits [kT]


# ---------------------------------------------------------------------- cases
def listed():
    return [
        # a 42 nm (17,0) tube at equilibrium, lowest two modes, ~115 energies: the smallest
        # call of a gate sweep, host arrays in and out (launches and latency count)
        dict(name="solve_small", kind="solve", m=17, cells=100, modes=2, eq="32 32 32", ne="", vds=0.0, mu=-1.0,
             pole_max=3.0, valence=-10.0, eta=1e-8, precision="fp64"),
        # an ordinary biased tube of an odd number of cells, the default contour (30 points
        # a path) and a 301-point bias window
        dict(name="solve_biased", kind="solve", m=17, cells=151, modes=3, eq="30 30 30", ne="301", vds=0.3, mu=0.0,
             pole_max=10.0, valence=-14.0, eta=1e-3, precision="fp64"),
        # a 6.8 um tube at few energies: few, very long recursions
        dict(name="solve_long", kind="solve", m=17, cells=16000, modes=2, eq="8 8 16", ne="64", vds=0.2, mu=0.0,
             pole_max=10.0, valence=-14.0, eta=1e-3, precision="fp64"),
        # the headline pass: 4000 sites, 8 modes, 4096 energies on device vectors
        dict(name="charge_full", kind="charge", m=17, cells=1000, modes=8, eq="256 256 512", ne="", window=3072,
             vds=0.5, mu=0.0, pole_max=10.0, valence=-14.0, eta=1e-4, precision="fp64"),
        # a 16-tube device of uneven lengths (200-2000 cells), 2-10 modes, 512-8192 energies
        dict(name="batch_fp64", kind="batch", tubes=16, spec=4, cells="200 2000", energies="512 8192", vds=0.4,
             precision="fp64"),
        # the same device in mixed precision with the broadened real axis in FP32
        dict(name="batch_mixed", kind="batch", tubes=16, spec=4, cells="200 2000", energies="512 8192", vds=0.4,
             precision="mixed"),
        # one gate point of a four-tube device, from zero charge to a 1e-4 residual
        dict(name="scf_point", kind="scf", tubes=4, spec=7, cells="60 300", energies="128 512", vds=0.4, vg=0.3,
             tol=1e-4),
        # real-space pass of 600 blocks of 26 atoms, ring-uniform potential
        dict(name="rs_ring", kind="rs", m=13, cells=300, eq="512 512 1024", ne="", vds=0.0, mu=-0.8, pole_max=3.0,
             eta=1e-6, atoms=False, precision="fp64"),
        # real-space pass with a potential per atom
        dict(name="rs_atoms", kind="rs", m=13, cells=75, eq="128 128 256", ne="", vds=0.0, mu=-0.8, pole_max=3.0,
             eta=1e-6, atoms=True, precision="fp64"),
        # a biased real-space pass of another chirality, per-atom potentials, mixed
        # precision (contour chains in FP32, the bias window in FP64)
        dict(name="rs_biased_mixed", kind="rs", m=10, cells=57, eq="64 64 128", ne="512", vds=0.3, mu=0.0,
             pole_max=3.0, eta=1e-3, atoms=True, precision="mixed"),
        # density of states, transmission, LDOS and current of a 1000-site tube
        dict(name="transport", kind="transport", m=17, cells=250, modes=4, ne="601", vds=0.3, mu=0.0, eta=2e-3),
        # one gradient of the operator on 4000 sites, batch 16
        dict(name="surrogate_grad", kind="train", sites=4000, batch=16),
    ]


def _ints(text):
    return [int(v) for v in text.split()]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "charge", "charge", "batch", "scf", "rs", "rs", "rs", "transport", "train"])
    mixed = rng.choice(["fp64", "fp64", "mixed"])
    vds = rng.choice([0.0, round(rng.uniform(0.05, 0.5), 3)])
    mu = -1.0 if vds == 0.0 else 0.0
    if kind in ("solve", "charge"):
        m = rng.choice([13, 17, 19])
        cells = _log(rng, 20, 8000)
        modes = rng.randint(1, m // 2 + 1)
        # at most about the work of charge_full
        budget = max(48, min(4096, int(1.2e8 / (4 * cells * modes))))
        total = _log(rng, 48, budget)
        q = max(4, total // 8 if vds else total // 4)
        eq = f"{q} {q} {2 * q}"
        ne = str(max(16, total - 4 * q)) if vds else ""
        return dict(kind=kind, m=m, cells=cells, modes=modes, eq=eq, ne=ne, vds=vds, mu=mu,
                    pole_max=3.0 if vds == 0.0 else 10.0, valence=-14.0, eta=rng.choice([5e-4, 1e-3, 2e-3]),
                    precision=mixed)
    if kind == "batch":
        lo = _log(rng, 30, 200)
        elo = _log(rng, 64, 512)
        return dict(kind="batch", tubes=rng.randint(2, 16), spec=rng.randrange(1 << 20), cells=f"{lo} {lo * 8}",
                    energies=f"{elo} {elo * 8}", vds=max(vds, 0.05), precision=mixed)
    if kind == "scf":
        lo = _log(rng, 20, 80)
        return dict(kind="scf", tubes=rng.randint(1, 6), spec=rng.randrange(1 << 20), cells=f"{lo} {lo * 4}",
                    energies="96 384", vds=round(rng.uniform(0.1, 0.5), 2), vg=round(rng.uniform(0.0, 0.6), 2), tol=1e-4)
    if kind == "rs":
        m = rng.randint(5, 16)
        cells = _log(rng, 6, 150)
        total = _log(rng, 64, max(96, min(1024, int(2.5e8 / (2 * cells * m ** 3)))))
        q = max(8, total // 8 if vds else total // 4)
        return dict(kind="rs", m=m, cells=cells, eq=f"{q} {q} {2 * q}", ne=str(max(16, total - 4 * q)) if vds else "", vds=vds,
                    mu=-0.8 if vds == 0.0 else 0.0, pole_max=3.0, eta=1e-3 if vds else 1e-6, atoms=rng.random() < 0.6,
                    precision=mixed)
    if kind == "transport":
        m = rng.choice([13, 17, 19])
        cells = _log(rng, 20, 500)
        return dict(kind="transport", m=m, cells=cells, modes=rng.randint(1, m // 2 + 1),
                    ne=str(_log(rng, 33, max(64, min(900, int(6e5 / (4 * cells)))))), vds=round(rng.uniform(0.1, 0.4), 3), mu=0.0,
                    eta=2e-3)
    return dict(kind="train", sites=8 * _log(rng, 40, 500), batch=rng.choice([4, 7, 8, 13, 16]))


# ---------------------------------------------------------------------- inputs
def _specs(case):
    """Descriptors of the tubes of a batch: chirality uniform, length, mode count and
    energy count spread as in an uneven multi-tube device."""
    r = np.random.default_rng(case["spec"])
    out = []
    for _ in range(case["tubes"]):
        m = int(r.choice([13, 17, 19]))
        cells = int(round(math.exp(r.uniform(*np.log(_ints(case["cells"]))))))
        modes = min(int(r.integers(2, 11)), m // 2 + 1)
        E = int(round(math.exp(r.uniform(*np.log(_ints(case["energies"]))))))
        q, h = max(2, E // 8), max(2, E // 4)
        ne = max(6, E - 2 * q - h)
        out.append(dict(m=m, cells=cells, modes=modes, eq=f"{q} {q} {h}",
                        ne=f"{ne // 4} {ne // 2} {ne - ne // 4 - ne // 2}", cuts=(30.0, 70.0), vds=case["vds"], mu=0.0, pole_max=10.0, valence=-14.0, eta=2e-3,
                        precision=case.get("precision", "fp64"), ra32=case.get("precision") == "mixed"))
    return out


def _tube_kwargs(s):
    kw = dict(type_id=(s["m"], 0), num_unitcells=s["cells"], num_modes=s.get("modes", 1),
              contact_mu=(s["mu"], s["mu"] - s["vds"]), contact_T=(300.0, 300.0),
              eq_integration_pts=tuple(_ints(s.get("eq", "30 30 30"))), E_pole_max=s.get("pole_max", 10.0),
              E_valence_min=s.get("valence", -14.0), E_zPlus_imag=s["eta"], precision=s.get("precision", "fp64"),
              mixed_realaxis_fp32=s.get("ra32", False))
    if s.get("window"):
        kw["realaxis_window"] = (-1.5, 1.5, s["window"], 0)
    if s.get("ne"):
        kw["noneq_integration_pts"] = tuple(_ints(s["ne"]))
    if s.get("cuts"):
        kw["noneq_percent_intercuts"] = s["cuts"]
    return kw


def _positions(cells):
    """Axial ring positions of a zigzag tube [nm]: four rings per cell."""
    base = np.array([1.0, 1.5, 2.5, 3.0]) * ACC
    y0 = -(cells / 2.0) * 3.0 * ACC - ACC / 2.0
    return (base[None, :] + 3 * ACC * np.arange(cells)[:, None] + y0).reshape(-1) / 1e-9


def _potential(cells, seed, amp=0.3, ramp=0.3):
    """Site potential [eV]: five Gaussian bumps (gates, impurities) and a drain ramp."""
    r = np.random.default_rng(seed)
    y = _positions(cells)
    L = y[-1] - y[0]
    U = ramp * (y - y[0]) / L
    for _ in range(5):
        U = U + r.uniform(-amp, amp) * np.exp(-((y - y[0] - r.uniform(0, L)) ** 2) / (2 * r.uniform(2.0, 10.0) ** 2))
    return U


def _atoms(case, U, seed):
    """Per-atom potential [N][m]: the ring value and 50 meV of disorder."""
    r = np.random.default_rng(seed + 17)
    return U[:, None] + 0.05 * r.standard_normal((len(U), case["m"]))


def _train_data(case, seed):
    S, B = case["sites"], case["batch"]
    r = np.random.default_rng(seed)
    x = np.arange(S) / S
    U = sum(r.uniform(-0.3, 0.3, (B, 1)) * np.exp(-((x[None, :] - r.uniform(0, 1, (B, 1))) ** 2) / 0.005) for _ in range(5))
    Vg, Vds = r.uniform(0, 0.8, B), r.uniform(0, 0.6, B)
    Y = np.tanh(3 * U) + 0.1 * Vg[:, None] * np.cos(6 * x)[None, :]
    return U.astype(np.float32), Vg.astype(np.float32), Vds.astype(np.float32), Y.astype(np.float32)


def prepare(case, seed):
    from electrostatic_b200.negf import CNT, ChargePlan
    kind = case["kind"]
    if kind in ("solve", "charge"):
        U = _potential(case["cells"], seed)
        st = dict(kind=kind, tube=CNT(**_tube_kwargs(case)), U=U, Uc=(float(U[0]), float(U[-1])))
        if kind == "charge":
            st["Ud"] = torch.tensor(U, device="cuda")
            st["Q"] = torch.zeros(len(U), dtype=torch.float64, device="cuda")
        return st
    if kind == "batch":
        tubes = []
        for i, s in enumerate(_specs(case)):
            t = CNT(**_tube_kwargs(s))
            U = _potential(s["cells"], seed + 100 * i)
            t.set_potential(U, (U[0], U[-1]))
            tubes.append(t)
        Q = torch.zeros(sum(t.num_field_sites for t in tubes), dtype=torch.float64, device="cuda")
        return dict(kind=kind, tubes=tubes, Q=Q, plan=ChargePlan(tubes, Q, autotune=True))
    if kind == "scf":
        from electrostatic_b200.scf import BatchSCF
        from electrostatic_b200.workloads import gate_with_contacts
        specs = _specs(case)
        tubes = [CNT(**_tube_kwargs(s)) for s in specs]
        gates = [gate_with_contacts(t.site_positions(), ACC * math.sqrt(3.0) * s["m"] / (2 * math.pi), vds=case["vds"])
                 for t, s in zip(tubes, specs)]
        scf = BatchSCF(tubes, gates, max_norm=case["tol"], fraction=0.1)
        r = np.random.default_rng(seed)
        U0 = []
        for g, s in zip(gates, specs):  # a gate point with a little disorder of its own
            y = _positions(s["cells"])
            bump = r.uniform(-0.05, 0.05) * np.exp(-((y - y.mean() * r.uniform(0.5, 1.5)) ** 2) / 18.0)
            U0.append(torch.tensor(g.external(case["vg"]) + bump, device="cuda"))
        return dict(kind=kind, scf=scf, tubes=tubes, gates=gates, U0=U0)
    if kind == "rs":
        U = _potential(case["cells"], seed, amp=0.2, ramp=0.2)
        t = CNT(**_tube_kwargs(case))
        t.set_potential(U, (U[0], U[-1]))
        Ua = torch.tensor(_atoms(case, U, seed), device="cuda") if case["atoms"] else None
        Q = torch.zeros(len(U), dtype=torch.float64, device="cuda")
        t.realspace_charge(out=Q, U_atoms=Ua)  # the tube's Rho0 is made by its first call and kept
        return dict(kind=kind, tube=t, Ua=Ua, Q=Q)
    if kind == "transport":
        U = _potential(case["cells"], seed)
        t = CNT(**_tube_kwargs(case))
        t.set_potential(U, (U[0], U[-1]))
        return dict(kind=kind, tube=t)
    from electrostatic_b200.surrogate import FourierOperator
    U, Vg, Vds, Y = _train_data(case, seed)
    op = FourierOperator(case["sites"], seed=seed % 1000)
    dev = [torch.tensor(a, device="cuda") for a in (U, Vg, Vds)]
    return dict(kind=kind, op=op, data=dev, Y=torch.tensor(Y.reshape(-1), device="cuda"), B=case["batch"])


def run(state):
    from electrostatic_b200.negf import compute_charge
    kind = state["kind"]
    if kind == "solve":
        return state["tube"].Solve_NEGF(state["U"], state["Uc"])
    if kind == "charge":
        state["tube"].set_potential_device(state["Ud"], state["Uc"])
        return compute_charge([state["tube"]], out=state["Q"])
    if kind == "batch":
        state["plan"].launch()
        return state["Q"]
    if kind == "scf":
        scf = state["scf"]
        scf.reset()
        scf.set_external(U0=state["U0"])
        steps, _ = scf.solve()
        return {"charge": scf.Q, "n_in": scf.n_in, "steps": steps}
    if kind == "rs":
        return state["tube"].realspace_charge(out=state["Q"], U_atoms=state["Ua"])
    if kind == "transport":
        d = state["tube"].Compute_DensityOfStates(ldos=True)
        return {"E": d["E"], "dos": d["dos"], "T": d["T"], "conductance": d["conductance"], "ldos": d["ldos"],
                "total": d["total_conductance"], "current": state["tube"].Compute_Current()}
    op, (U, Vg, Vds), B = state["op"], state["data"], state["B"]
    q = op.forward(op.features(U, Vg, Vds), B, keep=True)
    dq, part = op.loss_grad(q, state["Y"])
    op.backward(dq, B)
    return {"q": q, "loss": part, "grads": op.grads}


# ---------------------------------------------------------------------- work
def _counts(s):
    """(sites, modes, contour + pole energies, real-axis energies) of a mode-space pass."""
    it = _items(s)
    ra = int(np.sum(it["ra"]))
    return 4 * s["cells"], s["modes"], len(it["ra"]) - ra, ra


def work(case):
    """Operations with complex add 2, multiply 6, divide 11, |z|^2 3: 53 per contour and 76 per
    real-axis update of a site of a mode chain; 32 m^3 per ring-block update (an inversion and
    three products of complex m x m corners), 72 m^3 with the two contact columns.  Bytes: the
    potential, the charge and the energy table."""
    kind = case["kind"]
    if kind in ("solve", "charge", "batch", "scf"):
        b = f = 0.0
        for s in (_specs(case) if kind in ("batch", "scf") else [case]):
            N, M, c, r = _counts(s)
            f += N * M * (53.0 * c + 76.0 * r)
            b += 16.0 * N + 48.0 * (c + r)
        it = 12 if kind == "scf" else 1  # iterations from zero charge to the residual, about
        return {"bytes": b * it, "flops": f * it}
    if kind == "rs":
        it = _items(case)
        ra = int(np.sum(it["ra"]))
        c, m, K = len(it["ra"]) - ra, case["m"], 2 * case["cells"]
        if case["atoms"]:
            f = K * m ** 3 * (32.0 * c + 72.0 * ra)
        else:  # a ring-uniform potential decouples into the modes of the ring
            f = 2.0 * K * (m // 2 + 1) * (53.0 * c + 76.0 * ra)
        return {"bytes": 8.0 * 2 * K * (m if case["atoms"] else 1) + 16.0 * K + 48.0 * (c + ra), "flops": f}
    if kind == "transport":
        N, M, P = 4 * case["cells"], case["modes"], sum(_ints(case["ne"]))
        return {"bytes": 8.0 * N * (P + 1) + 48.0 * P, "flops": 76.0 * 2 * N * M * P}
    S, B, W, Md, L = case["sites"], case["batch"], 128, 32, 6
    R = S * B
    gemm = 2.0 * R * W * 24 + L * (2.0 * R * W * W + 2 * 2.0 * R * 2 * Md * W + 2.0 * B * Md * (2 * W) ** 2) + 2.0 * R * W
    params = 24 * W + W * 2 + 1 + L * (W * W + W + Md * 4 * W * W)
    return {"bytes": 4.0 * R * 2 + 4.0 * R + 6.0 * params, "flops": 3 * gemm}


# ---------------------------------------------------------------------- 64-bit reference
def _gauss_legendre(n):
    """Newton's method on P_n from cos(pi (i - 1/4) / (n + 1/2)), each node until its step is below
    3e-11 (the weights come from the last derivative: the scheme that defines the energy grids)."""
    x = np.cos(np.pi * (np.arange(1, (n + 1) // 2 + 1) - 0.25) / (n + 0.5))
    dp, live = np.ones_like(x), np.ones(len(x), bool)
    while live.any():
        z = x[live]
        p, pm = np.ones_like(z), np.zeros_like(z)
        for j in range(1, n + 1):
            p, pm = ((2 * j - 1) * z * p - (j - 1) * pm) / j, p
        d = n * (z * p - pm) / (z * z - 1)
        dp[live] = d
        x[live] = z - p / d
        live[live] = np.abs(p / d) > 3e-11
    w = 2.0 / ((1 - x * x) * dp * dp)
    k = n // 2
    return np.concatenate([-x, x[:k][::-1]]), np.concatenate([w, w[:k][::-1]])


def _line(a, b, n):
    x, w = _gauss_legendre(n)
    half = (b - a) * 0.5
    return half * x + (a + b) * 0.5, w * half


def _arc(a, b, n):
    x, w = _gauss_legendre(n)
    c = (b.real ** 2 - a.real ** 2 - a.imag ** 2) / (2 * (b.real - a.real))
    R = c - b.real
    t1 = math.asin(abs(a.imag) / R)
    if c > a.real:
        t1 = math.pi - t1
    th = (math.pi - t1) * 0.5 * x + (math.pi + t1) * 0.5
    return c + R * np.cos(th) + 1j * (b.imag + R * np.sin(th)), w * (math.pi - t1) * 0.5 * R * np.exp(1j * th) * 1j


def _fermi(z, kT):
    return 1.0 / (np.exp(z / kT) + 1.0)


def _contour(right, mu, kT, eta, eq, pole_max, valence):
    """The equilibrium contour below `right`: two lines and an arc, heights set by the poles."""
    n = int((pole_max - math.pi * kT) / (2 * math.pi * kT) + 1)
    zeta = complex(right.real, 2 * n * math.pi * kT)
    h = complex((mu if mu is not None else right.real) - TAIL * kT, zeta.imag)
    parts = [_line(right, zeta, eq[0]), _line(zeta, h, eq[1]), _arc(h, complex(valence, eta), eq[2])]
    return np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts]), n


def _items(s):
    """Energy points of a pass: E, coefficient c of Im(c G) (contour, poles), b0 and b1 of the two
    contacts' spectral functions (real axis), weights wJ of the real axis."""
    mu0, mu1 = s["mu"], s["mu"] - s["vds"]
    lo, hi, eta = min(mu0, mu1), max(mu0, mu1), s["eta"]
    kT = KB_EV * 300.0
    eq, window = _ints(s.get("eq", "30 30 30")), s.get("window")
    pole_max, valence = s.get("pole_max", 10.0), s.get("valence", -14.0)
    E, c, wr, Er = [], [], np.zeros(0, complex), np.zeros(0, complex)
    if s["vds"] == 0.0 and not window:
        Ec, wJ, n = _contour(complex(hi + TAIL * kT, eta), lo, kT, eta, eq, pole_max, valence)
        poles = lo + 1j * math.pi * kT * (2 * np.arange(n) + 1)
        E += [Ec, poles]
        c += [(-2.0 / math.pi) * wJ * _fermi(Ec - lo, kT), np.full(n, -4j * kT)]
    else:
        right = complex(-1.5 if window else lo - TAIL * kT, eta)
        last = complex(1.5 if window else hi + TAIL * kT, eta)
        Ec, wJ, _ = _contour(right, None, kT, eta, eq, pole_max, valence)
        E.append(Ec)
        c.append((-2.0 / math.pi) * wJ * _fermi(Ec - lo, kT))
        if window:
            dE = (last - right) / (window - 1)
            Er, wr = right + np.arange(window) * dE, np.full(window, dE)
        else:
            ne = _ints(s["ne"])
            cuts = [0.0] + list(s.get("cuts") or [(p + 1) * 100.0 / len(ne) for p in range(len(ne) - 1)]) + [100.0]
            ends = [right + (q / 100.0) * (last - right) for q in cuts]
            parts = [_line(ends[p], ends[p + 1], n) for p, n in enumerate(ne)]
            Er, wr = np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])
    E, c = np.concatenate(E), np.concatenate(c)
    b = [((-1.0 / math.pi) * wr * _fermi(Er - mu, kT)).real for mu in (mu0, mu1)]
    z = np.zeros(len(E))
    return dict(E=np.concatenate([E, Er]), c=np.concatenate([c, 0 * Er]), b0=np.concatenate([z, b[0]]),
                b1=np.concatenate([z, b[1]]), ra=np.concatenate([z > 1, np.ones(len(Er), bool)]), Er=Er, wr=wr,
                f=[_fermi(Er - mu, kT) for mu in (mu0, mu1)])


def _rho0_items(s):
    kT, eta = KB_EV * 300.0, s["eta"]
    E, wJ, _ = _contour(complex(TAIL * kT, eta), 0.0, kT, eta, (30, 30, 30), s.get("pole_max", 10.0),
                        s.get("valence", -14.0))
    # the first line starts at the origin
    n = int((s.get("pole_max", 10.0) - math.pi * kT) / (2 * math.pi * kT) + 1)
    zeta = complex(TAIL * kT, 2 * n * math.pi * kT)
    E[:30], wJ[:30] = _line(complex(0.0, eta), zeta, 30)
    z = np.zeros(len(E))
    return dict(E=E, c=(-2.0 / math.pi) * wJ, b0=z, b1=z, ra=z > 1)


def _modes(m, count):
    """(beta_J, degeneracy) of the lowest `count` distinct modes of an (m,0) tube."""
    gap = {p: min(abs(3 * p - 2 * m), abs(3 * p - m)) for p in range(1, m + 1)}
    out = []
    for g in sorted(set(gap.values())):
        ps = [p for p in gap if gap[p] == g]
        out.append((2 * GAMMA * math.cos(math.pi * ps[0] / m), float(len(ps))))
    return out[:count]


def _ring_modes(m):
    """(beta_k, multiplicity) of the Fourier modes of a ring of m atoms."""
    return [(2 * GAMMA * math.cos(math.pi * k / m), 1.0 if k == 0 or 2 * k == m else 2.0) for k in range(m // 2 + 1)]


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _surface(E, beta):
    """Surface Green's function of a lead of alternating hoppings, retarded root."""
    F = E * E + GAMMA ** 2 - beta * beta
    S = torch.sqrt(F * F - 4 * GAMMA ** 2 * E * E)
    D = 2 * GAMMA ** 2 * E
    a, b = (F + S) / D, (F - S) / D
    return torch.where(a.imag < 0, a, torch.where(b.imag < 0, b, torch.zeros_like(a)))


def _mode_pass(U, modes, it, per_site):
    """Scalar recursions of every (mode, energy) chain; per_site(n, G, lam, rho, chain data) takes
    the site values.  lam, rho: running products of the contacts' columns.  it["on"] is 1 for the
    chains that see the potential U and 0 for those of the U = 0 pass."""
    dev = _dev()
    N = len(U)
    t = lambda a, d: torch.tensor(np.asarray(a), dtype=d, device=dev)
    M, P = len(modes), len(it["E"])
    beta = t(np.repeat([b for b, _ in modes], P), torch.float64)
    deg = t(np.repeat([d for _, d in modes], P), torch.float64)
    E = t(np.tile(it["E"], M), torch.complex128)
    on = t(np.tile(it["on"], M), torch.float64)
    ch = dict(c=t(np.tile(it["c"], M), torch.complex128) * deg, deg=deg)
    S0 = GAMMA ** 2 * _surface(E - U[0] * on, beta)
    S1 = GAMMA ** 2 * _surface(E - U[-1] * on, beta)
    ch["g0"], ch["g1"] = -2 * S0.imag, -2 * S1.imag
    ch["k0"] = ch["g0"] * deg * t(np.tile(it["b0"], M), torch.float64)
    ch["k1"] = ch["g1"] * deg * t(np.tile(it["b1"], M), torch.float64)
    h2 = [beta * beta, torch.full_like(beta, GAMMA ** 2)]
    C = E.numel()
    Y = torch.zeros(N, C, dtype=torch.complex128, device=dev)
    lam = torch.ones(N, C, dtype=torch.float64, device=dev)
    for n in range(N - 1):
        a = E - U[n] * on
        if n == 0:
            a = a - S0
        g = 1.0 / (a - Y[n])
        torch.mul(g, h2[n & 1], out=Y[n + 1])
        torch.mul(lam[n], h2[n & 1] * (g.real ** 2 + g.imag ** 2), out=lam[n + 1])
    X = torch.zeros_like(E)
    rho = torch.ones_like(beta)
    for n in range(N - 1, -1, -1):
        a = E - U[n] * on
        if n == 0:
            a = a - S0
        if n == N - 1:
            a = a - S1
        per_site(n, 1.0 / (a - X - Y[n]), lam[n], rho, ch)
        if n:
            g = 1.0 / (a - X)
            X = h2[(n - 1) & 1] * g
            rho = rho * h2[(n - 1) & 1] * (g.real ** 2 + g.imag ** 2)


def _tube_exact(s, U, modes, rho0_only=False):
    """Charge per site: the pass at U (left out with rho0_only) minus the pass at U = 0."""
    it, r0 = _items(s), _rho0_items(s)
    r0["c"] = -r0["c"]
    both = [dict(r0, on=np.zeros(len(r0["E"])))] + ([] if rho0_only else [dict(it, on=np.ones(len(it["E"])))])
    it = {k: np.concatenate([d[k] for d in both]) for k in ("E", "c", "b0", "b1", "on")}
    Q = torch.zeros(len(U), dtype=torch.float64, device=_dev())

    def site(n, G, lam, rho, ch):
        Q[n] += ((ch["c"] * G).imag + (G.real ** 2 + G.imag ** 2) * (lam * ch["k0"] + rho * ch["k1"])).sum()
    step = max(1, int(3e10 / (24.0 * len(U) * len(modes))))  # up to 30 GB of Y and lam at a time
    for i in range(0, len(it["E"]), step):
        _mode_pass(U, modes, {k: v[i:i + step] for k, v in it.items()}, site)
    return Q.cpu().numpy()


def _rs_atoms_exact(case, U, Ua):
    """Ring-by-ring matrix recursions (m x m) with a potential per atom."""
    dev, m, N = _dev(), case["m"], len(U)
    it = _items(case)
    g = GAMMA
    C = np.zeros((m, m))
    for j in range(m):
        C[j, j] += 1.0
        C[j, (j + 1) % m] += 1.0
    hop = [torch.tensor(g * C, dtype=torch.complex128, device=dev), g * torch.eye(m, dtype=torch.complex128, device=dev)]
    k = np.arange(m)
    Fk = torch.tensor(np.exp(2j * np.pi * np.outer(k, k) / m) / math.sqrt(m), device=dev)
    beta = torch.tensor(2 * g * np.cos(np.pi * k / m), device=dev)
    Ut = torch.tensor(Ua, device=dev)

    def lead(E, u):
        s = _surface(E[:, None] - u, beta[None, :])
        return torch.einsum("jk,ek,lk->ejl", Fk, s, Fk.conj())

    def sums(E, c, b0, b1, ra):
        Et = torch.tensor(E, device=dev)
        sL, sR = g * g * lead(Et, U[0]), g * g * lead(Et, U[-1])
        I = torch.eye(m, dtype=torch.complex128, device=dev)

        def alpha(n):
            return Et[:, None, None] * I - torch.diag(Ut[n].to(torch.complex128))[None]
        SL, B = [sL], None
        if ra:
            ident = I.expand(len(E), m, m)
            B = [ident]
        for n in range(N - 1):
            gl = torch.linalg.inv(alpha(n) - SL[n])
            T = hop[n & 1]
            SL.append(T.T @ gl @ T)
            if ra:
                B.append(T.T @ (gl @ B[n]))
        SR, D = sR, I.expand(len(E), m, m)
        out = torch.zeros(N, dtype=torch.float64, device=dev)
        ct = torch.tensor(c, device=dev)
        if ra:
            GL, GR = [1j * (x - x.conj().transpose(1, 2)) for x in (sL, sR)]
            w0, w1 = torch.tensor(b0, device=dev), torch.tensor(b1, device=dev)
        for n in range(N - 1, -1, -1):
            a = alpha(n)
            G = torch.linalg.inv(a - SL[n] - SR)
            if ra:
                L, R = G @ B[n], G @ D
                A0 = torch.einsum("eij,ejk,eik->e", L, GL, L.conj()).real
                A1 = torch.einsum("eij,ejk,eik->e", R, GR, R.conj()).real
                out[n] += (w0 * A0 + w1 * A1).sum()
            else:
                out[n] += (ct * torch.diagonal(G, dim1=1, dim2=2).sum(1)).imag.sum()
            if n:
                gr = torch.linalg.inv(a - SR)
                T = hop[(n - 1) & 1]
                if ra:
                    D = T @ (gr @ D)
                SR = T @ gr @ T.T
        return out

    Q = torch.zeros(N, dtype=torch.float64, device=dev)
    step = max(8, int(8e9 / (32.0 * N * m * m)))
    for kind in (False, True):
        idx = np.nonzero(it["ra"] == kind)[0]
        for i in range(0, len(idx), step):
            j = idx[i:i + step]
            Q += sums(it["E"][j], it["c"][j], it["b0"][j], it["b1"][j], kind)
    return Q.cpu().numpy() + _tube_exact(case, 0 * U, _ring_modes(m), rho0_only=True)


def _transport_exact(case, U):
    it = _items(case)
    keep = it["ra"]
    part = dict({k: it[k][keep] for k in ("E", "c", "b0", "b1")}, on=np.ones(int(keep.sum())))
    N, P, M = len(U), int(keep.sum()), case["modes"]
    ldos = torch.zeros(N, P, dtype=torch.float64, device=_dev())
    T = {}

    def site(n, G, lam, rho, ch):
        g2 = G.real ** 2 + G.imag ** 2
        a, b = ch["deg"] * ch["g0"] * g2 * lam, ch["deg"] * ch["g1"] * g2 * rho
        ldos[n] = (a + b).reshape(M, P).sum(0)
        if n == 0:
            T[0] = (ch["g0"] * b).reshape(M, P).sum(0)
        if n == N - 1:
            T[1] = (ch["g1"] * a).reshape(M, P).sum(0)
    _mode_pass(U, _modes(case["m"], M), part, site)
    E, Er = it["Er"], it["Er"].real
    T0, T1 = T[0].cpu().numpy(), T[1].cpu().numpy()
    dos = 2.0 * ldos.sum(0).cpu().numpy() / (2 * math.pi) / (4 * case["m"])
    dE = Er[0] - Er[1]
    F = _fermi(Er - case["mu"], KB_EV * 300.0)
    dF = np.empty(P)
    dF[1:-1] = F[2:] - F[:-2]
    dF[0], dF[-1] = -3 * F[0] + 4 * F[1] - F[2], 3 * F[-1] - 4 * F[-2] + F[-3]
    cond = -T0 * dF / (2 * dE)
    cm = 2.0 * Q_E / H_EV
    w = (it["f"][0] - it["f"][1]) * it["wr"]
    I = np.array([np.sum((cm * w).real * T0), np.sum((-cm * w).real * T1)])
    return {"E": E, "dos": dos, "T": T0, "conductance": cond, "ldos": (ldos / (2 * math.pi)).T.cpu().numpy(),
            "total": float(np.sum(cond * dE)), "current": I}


def _train_exact(case, seed):
    """The operator and its gradient in 64 bits from the same (BF16) weights and features."""
    from torch.nn import functional as Fn
    dev, S, B = _dev(), case["sites"], case["batch"]
    W, Md, L, feat, win = 128, 32, 6, 24, 8
    gen = torch.Generator().manual_seed(seed % 1000)

    def init(shape, fan):
        return torch.randn(*shape, generator=gen, dtype=torch.float32) / math.sqrt(fan)
    p = {"W_lift": init((feat, W), feat), "b_lift": torch.zeros(W), "w_p": init((W,), W), "b_p": torch.zeros(1)}
    for l in range(L):
        p[f"W{l}"], p[f"R{l}"], p[f"b{l}"] = init((W, W), W), init((Md, 2 * W, 2 * W), 2 * W) * 0.5, torch.zeros(W)
    p = {k: (v if k in ("w_p",) or k.startswith("b") else v.to(torch.bfloat16)).double().to(dev).requires_grad_() for k, v in p.items()}
    U, Vg, Vds, Y = _train_data(case, seed)
    n = np.arange(S)
    j = n[:, None] + np.arange(-win, win + 1)[None, :]
    x = np.zeros((B, S, feat), dtype=np.float32)
    x[:, :, :17] = U[:, np.clip(j, 0, S - 1)] * ((j >= 0) & (j < S)).astype(np.float32)
    x[:, :, 17], x[:, :, 18] = Vg[:, None], Vds[:, None]
    x[:, :, 19], x[:, :, 20] = n / S, np.where(n % 2 == 0, 1.0, -1.0)
    x[:, :, 21], x[:, :, 22] = np.exp(-n / 40.0), np.exp(-(S - 1 - n) / 40.0)
    x = torch.tensor(x).to(torch.bfloat16).double().to(dev)
    ang = 2 * np.pi * np.outer(np.arange(Md), n) / S
    G = np.stack([np.cos(ang), np.sin(ang)], 1).reshape(2 * Md, S)
    F = 2.0 / S * G
    F[0] *= 0.5
    F, G = (torch.tensor(a, dtype=torch.bfloat16).double().to(dev) for a in (F, G.T.copy()))
    h = x @ p["W_lift"] + p["b_lift"]
    for l in range(L):
        hat = torch.einsum("ks,bsw->bkw", F, h).reshape(B, Md, 2 * W)
        z = torch.einsum("bki,kij->bkj", hat, p[f"R{l}"]).reshape(B, 2 * Md, W)
        h = Fn.gelu(h @ p[f"W{l}"] + torch.einsum("sk,bkw->bsw", G, z) + p[f"b{l}"], approximate="tanh")
    q = (h @ p["w_p"] + p["b_p"]).reshape(-1)
    y = torch.tensor(Y.reshape(-1)).double().to(dev)
    sq = (q - y) ** 2
    sq.mean().backward()
    loss = Fn.pad(sq, (0, -len(sq) % 256)).reshape(-1, 256).sum(1)
    return {"q": q.detach().cpu().numpy(), "loss": loss.detach().cpu().numpy(),
            "grads": {k: v.grad.cpu().numpy() for k, v in p.items()}}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "charge"):
        return _tube_exact(case, _potential(case["cells"], seed), _modes(case["m"], case["modes"]))
    if kind == "batch":
        return np.concatenate([_tube_exact(s, _potential(s["cells"], seed + 100 * i), _modes(s["m"], s["modes"]))
                               for i, s in enumerate(_specs(case))])
    if kind == "rs":
        U = _potential(case["cells"], seed, amp=0.2, ramp=0.2)
        if case["atoms"]:
            return _rs_atoms_exact(case, U, _atoms(case, U, seed))
        return _tube_exact(case, U, _ring_modes(case["m"]))
    if kind == "transport":
        return _transport_exact(case, _potential(case["cells"], seed))
    if kind == "train":
        return _train_exact(case, seed)
    return None  # a self-consistent solve has no closed value
