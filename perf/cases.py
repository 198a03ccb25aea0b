"""The work that a user of this framework has it do, as measurable cases.

The framework runs FORGE's self-consistent Hartree-Fock loop for twisted multilayer graphene, so
most cases are one SCF iteration (assembly of every H(k), the batched partial eigen-solve, Fermi
level, density matrix, energies, mixing, potential) over the sizes of this repository's
configurations and tests: (m, m+1) bilayers from m = 2 (the smoke test) to m = 20 (N = 5044),
plain FP64 and mixed precision with the eigenpair refinement (the benchmark's fast path), OptimalStep
and Pulay mixing.  The others are the calls around it: the bands alone, several systems of
different size in one group, the allocation-free eigen-solver on a caller's device matrix, the
gradient of the warm-start network and the long-range Hartree kernel of a new system.

The starting state of an iteration is a field of the kind the warm start predicts (site
densities and the density matrix on short bonds), made from the seed.
"""
import ctypes
import math

import numpy as np
import torch

import forge_gb300 as fg
from forge_gb300 import warmstart

# constants of the model (Setup.f90): lattice constant units, eV
A0, R0, D0, XI = 1.0 / math.sqrt(3.0), 0.184, 1.35772, 10.0 / 0.246
HUBBARD_U, ENERGY_TOL = 4.0, 1e-4
ROTATE = {2: (-1, 1), 3: (-1, 1, -1)}


def listed():
    return [
        # the smallest self-consistent run (the smoke test's cell): launches and latency count
        scf("scf_fp64_m2_k3", 2, 3),
        # the regression configuration: a (5,6) bilayer, 6 x 6 k, neutrality, reference rules
        scf("scf_fp64_m5_k6", 5, 6),
        # the production-like parity cell, plain FP64 with Pulay mixing, nu = +2
        scf("scf_fp64_m10_k4", 10, 4, mixing="pulay", nfilling=2.0, deg="corrected"),
        # a large cell in plain FP64 at one k point
        scf("scf_fp64_m16_k1", 16, 1, nfilling=2.0, deg="corrected"),
        # the benchmark's fast path (mixed precision, every eigenpair refined, Pulay) from a small ...
        scf("scf_refined_m5_k6", 5, 6, mixed=True, mixing="pulay", deg="corrected"),
        # ... over the parity cell ...
        scf("scf_refined_m10_k4", 10, 4, mixed=True, mixing="pulay", nfilling=2.0, deg="corrected"),
        # ... to a magic-angle-sized one
        scf("scf_refined_m20_k1", 20, 1, mixed=True, mixing="pulay", nfilling=2.0, deg="corrected"),
        # band energies alone from the mixed solver (band plots at a given field)
        {"name": "bands_mixed_m12_k3", "kind": "bands", "ntheta": 12, "nlayers": 2, "numk": 3, "mixed": True,
         "nfilling": 0.0, "deg": "corrected"},
        # training-set generation: systems of different size share one eigen-solve
        {"name": "group_fp64_m3_m4_m5", "kind": "group", "m0": 3, "m1": 4, "m2": 5, "numk": 3, "nfilling": 0.0,
         "deg": "corrected"},
        # zdiagRed on a caller's device matrix (odd size) without allocation
        {"name": "zheevr_noalloc_n257", "kind": "zheevr", "n": 257, "iu": 139},
        # one training step's gradient of the bond network (BF16 weights) on a cell's bonds
        {"name": "mlp_gradient_14560", "kind": "mlp", "din": 18, "dout": 2, "batch": 14560},
        # the long-range Hartree kernel of a new system
        {"name": "long_range_m10", "kind": "long_range", "ntheta": 10, "nlayers": 2},
    ]


def scf(name, ntheta, numk, nlayers=2, mixed=False, mixing="oda", nfilling=0.0, deg="reference"):
    return {"name": name, "kind": "scf", "ntheta": ntheta, "nlayers": nlayers, "numk": numk, "mixed": mixed,
            "mixing": mixing, "nfilling": nfilling, "deg": deg}


def ndim(ntheta, nlayers):
    return nlayers * 2 * (3 * ntheta * ntheta + 3 * ntheta + 1)


def draw(rng):
    kind = rng.choices(["scf", "refined", "bands", "group", "zheevr", "mlp", "long_range"],
                       [6, 4, 2, 1, 2, 1, 1])[0]
    fill = rng.choice([-3.0, -2.0, -1.0, 0.0, 1.0, 2.0, 3.0])
    if kind == "zheevr":
        n = int(round(math.exp(rng.uniform(math.log(24), math.log(512)))))
        return {"kind": "zheevr", "n": n, "iu": rng.randint(max(1, n // 4), n)}
    if kind == "mlp":
        din, dout = rng.choice([(12, 1), (18, 2)])
        return {"kind": "mlp", "din": din, "dout": dout,
                "batch": int(round(math.exp(rng.uniform(math.log(300), math.log(40000)))))}
    if kind == "group":
        m = rng.randint(1, 5)
        return {"kind": "group", "m0": m, "m1": m + 1, "m2": m + 2, "numk": rng.randint(1, 3), "nfilling": fill,
                "deg": "corrected"}
    nlayers = rng.choice([2, 2, 2, 3])
    top = {"scf": 13 if nlayers == 2 else 10, "refined": 19 if nlayers == 2 else 15,
           "bands": 16 if nlayers == 2 else 12, "long_range": 14 if nlayers == 2 else 11}[kind]
    ntheta = int(round(math.exp(rng.uniform(math.log(2), math.log(top)))))
    if kind == "long_range":
        return {"kind": "long_range", "ntheta": ntheta, "nlayers": nlayers}
    # as many k points as keep the pass below the largest listed one's cost
    n = ndim(ntheta, nlayers)
    most = {"scf": 2.4e10, "refined": 4e10, "bands": 6e10}[kind] / float(n) ** 3
    numk = rng.randint(1, max(1, min(7, int(math.sqrt(most)))))
    if kind == "bands":
        return {"kind": "bands", "ntheta": ntheta, "nlayers": nlayers, "numk": numk, "mixed": rng.random() < 0.7,
                "nfilling": fill, "deg": "corrected"}
    c = scf("", ntheta, numk, nlayers, kind == "refined", "pulay" if kind == "refined" else rng.choice(["oda", "pulay"]),
            fill, "corrected")
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _setup(ntheta, nlayers, numk, mixed, nfilling, deg, xi=XI):
    return fg.Setup(ntheta=ntheta, nlayers=nlayers, RotateLayers=ROTATE[nlayers], numk=numk, nfilling=nfilling,
                    degfactor_mode=deg, precision="mixed" if mixed else "fp64", xi=xi)


def _gated(case, seed):
    """The set-up of a long-range case: the gate distance comes from the seed."""
    xi = XI * (0.8 + 0.4 * ((seed * 2654435761) % 65536) / 65536.0)
    return _setup(case["ntheta"], case["nlayers"], 1, False, 0.0, "corrected", xi)


def _cells(geo):
    """The translations R_c of the four stored cells, (4, 2)."""
    n1, n2 = np.asarray(geo.nUnitCell_1, float), np.asarray(geo.nUnitCell_2, float)
    t = np.asarray(geo.tn)
    return n1[:, None] * t[None, :, 0] + n2[:, None] * t[None, :, 1]


def _field(geo, nfilling, seed):
    """A predicted field: T[c, j, i] = P_ij(R_c) on bonds shorter than 1.6 a, densities near one half."""
    X = torch.as_tensor(np.ascontiguousarray(geo.Coords), device="cuda")
    n, gen = X.shape[0], _gen(seed)
    u = torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
    amp = torch.randn(2, generator=gen, device="cuda", dtype=torch.float64)
    T = torch.zeros(4, n, n, dtype=torch.complex128, device="cuda")
    for c, R in enumerate(_cells(geo)):
        dx = X[None, :, 0] - (X[:, None, 0] - R[0])
        dy = X[None, :, 1] - (X[:, None, 1] - R[1])
        dz = X[None, :, 2] - X[:, None, 2]
        d = torch.sqrt(dx * dx + dy * dy + dz * dz)
        plane = dz.abs() < 0.1
        b = torch.where(plane, 0.26 * torch.exp(-((d - A0) / 0.15) ** 2) - 0.08 * torch.exp(-((d - 2 * A0) / 0.15) ** 2),
                        0.04 * torch.exp(-((d - D0) / 0.2) ** 2))
        b = torch.where((d < 1.6) & (d > 0.1), b, torch.zeros_like(b))
        T[c] = torch.complex(b * (1 + 0.02 * (u[None, :] + u[:, None])), b * 0.01 * (u[None, :] - u[:, None]))
    g = torch.as_tensor(np.stack([geo.g1, geo.g12]), device="cuda")
    wave = torch.cos(X[:, :2] @ g.T) @ (0.002 + 0.0005 * amp)
    dens = 0.5 + nfilling / (2.0 * n) + wave - wave.mean() + 1e-4 * (u - u.mean())
    i = torch.arange(n, device="cuda")
    T[0, i, i] = dens.to(torch.complex128)
    return T


def _matrix(case, seed):
    """A seeded Hermitian matrix with a band-like spectrum of a few eV (lower triangle used)."""
    n, gen = case["n"], _gen(seed)
    a = torch.randn(n, n, generator=gen, device="cuda", dtype=torch.complex128)
    return (a + a.mH) / (2.0 * math.sqrt(n)) * 4.0


def _mlp_inputs(case, seed):
    gen, din, dout, n = _gen(seed), case["din"], case["dout"], case["batch"]
    shapes = ((128, din), (128,), (128, 128), (128,), (128, 128), (128,), (dout, 128), (dout,))
    p = torch.cat([(torch.rand(*s, generator=gen, device="cuda") * 2 - 1).reshape(-1) *
                   (math.sqrt(3.0 / s[-1]) if len(s) > 1 else 0.1) for s in shapes])
    x = torch.randn(n, din, generator=gen, device="cuda").clamp(-3, 3)
    y = torch.randn(n, dout, generator=gen, device="cuda") * 0.3
    return p.cpu().numpy(), x.cpu().numpy(), y.cpu().numpy(), shapes


def _context(ntheta, nlayers, numk, mixed, mixing, nfilling, deg, seed):
    S = _setup(ntheta, nlayers, numk, mixed, nfilling, deg)
    geo = fg.build_geometry(S)
    hf = fg.HartreeFock(S, geo)
    hf.LongRangeInteraction(copy_out=False)
    if mixing == "pulay":
        hf.set_mixing("pulay", depth=6, beta=0.7)
    if mixed and mixing:
        hf.set_eigen_refinement(1)
    hf.SetState(_field(geo, nfilling, seed).cpu().numpy().transpose(2, 1, 0))
    return {"hf": hf, "E": hf.PrepareState(), "out": _host_state(hf.N)}


def _host_state(n):
    """The host arrays that a driver keeps for the state: zFock, densities, potential (pinned)."""
    P = torch.empty(4 * n * n, dtype=torch.complex128, pin_memory=True).numpy().reshape(4, n, n)
    return P, np.empty(n), np.empty(n)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "scf":
        return dict(_context(case["ntheta"], case["nlayers"], case["numk"], case["mixed"], case["mixing"],
                             case["nfilling"], case["deg"], seed), kind=kind)
    if kind == "bands":
        return dict(_context(case["ntheta"], case["nlayers"], case["numk"], case["mixed"], "", case["nfilling"],
                             case["deg"], seed), kind=kind)
    if kind == "group":
        parts = [_context(case[m], 2, case["numk"], False, "oda", case["nfilling"], case["deg"], seed + 7 * q)
                 for q, m in enumerate(("m0", "m1", "m2"))]
        return {"kind": kind, "hf": [p["hf"] for p in parts], "E": np.array([p["E"] for p in parts]),
                "out": [p["out"] for p in parts]}
    if kind == "zheevr":
        H = _matrix(case, seed)
        lib = fg.load_library()
        f = lib.forge_gpu_zheevr_noalloc
        f.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_int64] + [ctypes.c_void_p] * 3
        f.restype = ctypes.c_int
        n, iu = case["n"], case["iu"]
        return {"kind": kind, "f": f, "n": n, "iu": iu, "H": H, "A": torch.empty_like(H),
                "w": torch.empty(iu, dtype=torch.float64, device="cuda"),
                "Z": torch.empty(iu, n, dtype=torch.complex128, device="cuda")}
    if kind == "mlp":
        p, x, y, _ = _mlp_inputs(case, seed)
        net = warmstart.Mlp(case["din"], case["dout"], 1)
        lib = fg.load_library()
        lib.forge_gpu_mlp_set_params(net.h, p.ctypes.data_as(ctypes.c_void_p))
        return {"kind": kind, "net": net, "x": x, "y": y, "g": np.empty_like(p), "loss": np.empty(1, np.float32)}
    if kind == "long_range":
        return {"kind": kind, "hf": fg.HartreeFock(_gated(case, seed))}
    raise ValueError(kind)


# ------------------------------------------------------------------------------------------- one pass
def _state(hf, out):
    P, d, V = out
    rc = hf.lib.forge_gpu_get_state(hf.ctx, P.ctypes.data_as(ctypes.c_void_p), d.ctypes.data_as(ctypes.c_void_p),
                                    V.ctypes.data_as(ctypes.c_void_p))
    if rc:
        raise RuntimeError("get_state: %d" % rc)
    return {"P": P, "density": d, "potential": V}


def _report(rep, E):
    return {"energies": np.array(E), "total": np.array([rep["TotalEnergyIn"], rep["TotalEnergy"]]),
            "fermi": np.array([rep["FermiEnergy"]]), "step": float(rep["Step"]), "residual": float(rep["residual"]),
            "density_change": float(rep["DensityConvergence"]),
            "counts": np.array([rep["nFermiLevel"], rep["nOccStates"], rep["nPartOccStates"], rep["info"]])}


def run(state):
    kind = state["kind"]
    if kind == "scf":
        hf = state["hf"]
        rep, state["E"], _ = hf.ScfIteration(state["E"])
        return dict(_report(rep, state["E"]), **_state(hf, state["out"]), bands=hf.GetBands())
    if kind == "bands":
        bands, _, _, info = state["hf"].Solve()
        return {"bands": bands, "info": info}
    if kind == "group":
        reps, state["E"], _ = fg.ScfIterationGroup(state["hf"], state["E"])
        return [dict(_report(r, e), **_state(hf, o)) for r, e, hf, o in zip(reps, state["E"], state["hf"], state["out"])]
    if kind == "zheevr":
        # the solver overwrites its matrix: a caller hands over a fresh one each time
        state["A"].copy_(state["H"])
        stream = torch.cuda.current_stream().cuda_stream
        rc = state["f"](state["A"].data_ptr(), state["n"], state["iu"], state["w"].data_ptr(), state["Z"].data_ptr(),
                        stream)
        return {"info": rc, "w": state["w"], "Z": state["Z"]}
    if kind == "mlp":
        net = state["net"]
        rc = net.lib.forge_gpu_mlp_gradient(net.h, *[state[k].ctypes.data_as(ctypes.c_void_p) for k in ("x", "y")],
                                            state["x"].shape[0],
                                            *[state[k].ctypes.data_as(ctypes.c_void_p) for k in ("g", "loss")])
        return {"rc": rc, "gradient": state["g"], "loss": float(state["loss"][0])}
    return {"LR": state["hf"].LongRangeInteraction()}


# ------------------------------------------------------------------------------------------- what a pass cannot do without
def _scf_work(n, nk, forms=True):
    iu = n / 2 + 10
    flops = nk * (16.0 / 3.0 * n ** 3 + 8.0 * n * n * iu)
    if forms:
        flops += nk * 4.0 * n * n * (n / 2)
    # tables and P read once, P written once
    return {"bytes": n * n * (25 * 8.0 + 64.0 + (64.0 if forms else 0.0)), "flops": flops}


def work(case):
    kind = case["kind"]
    if kind in ("scf", "bands"):
        return _scf_work(float(ndim(case["ntheta"], case["nlayers"])), case["numk"] ** 2, kind == "scf")
    if kind == "group":
        w = [_scf_work(float(ndim(case[m], 2)), case["numk"] ** 2) for m in ("m0", "m1", "m2")]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    if kind == "zheevr":
        n, iu = float(case["n"]), float(case["iu"])
        return {"bytes": 16.0 * n * (n / 2 + iu) + 8 * iu, "flops": 16.0 / 3.0 * n ** 3 + 8.0 * n * n * iu}
    if kind == "mlp":
        p = 128.0 * (case["din"] + 256 + case["dout"])
        return {"bytes": 4.0 * case["batch"] * (case["din"] + case["dout"]) + 6.0 * p, "flops": 6.0 * case["batch"] * p}
    n = float(ndim(case["ntheta"], case["nlayers"]))
    # 37 cells of 41 images, about eight operations each, on half the pairs
    return {"bytes": 8.0 * n * n, "flops": n * n / 2 * 37 * 41 * 8}


# ------------------------------------------------------------------------------------------- the same in plain 64-bit torch
def _ft(xi, yi, zi, xj, yj, zj):
    dx, dy, dz = xi - xj, yi - yj, zi - zj
    r = torch.sqrt(dx * dx + dy * dy + dz * dz)
    ok = r > 0.001
    r = torch.where(ok, r, torch.ones_like(r))
    cs2 = (dz / r) ** 2
    return torch.where(ok, -2.7 * torch.exp((A0 - r) / R0) * (1 - cs2) + 0.48 * torch.exp((D0 - r) / R0) * cs2,
                       torch.zeros_like(r))


def _fv(xi, yi, zi, xj, yj, zj, nlayers, gate):
    """The dual-gate screened interaction (41 images near, exponential far)."""
    rho2 = (xi - xj) ** 2 + (yi - yj) ** 2
    rho = torch.sqrt(rho2)
    v = torch.zeros_like(rho2)
    for n in range(-20, 21):
        sg = -1.0 if n % 2 else 1.0
        # the n = 0 image of a site on itself is excluded below
        v = v + sg / torch.sqrt(rho2 + (zj - (n * gate + zi * sg)) ** 2)
    far = 2.0 * math.sqrt(2.0) / torch.sqrt(rho / gate) * torch.exp(-math.pi * rho / gate) / gate
    v = torch.where((rho < gate) | (rho < 2 * nlayers * D0), v, far)
    return torch.where(rho2 + (zi - zj) ** 2 > 1e-4, v, torch.zeros_like(v))


def _xyz(geo):
    X = torch.as_tensor(np.ascontiguousarray(geo.Coords), device="cuda")
    return X[:, 0], X[:, 1], X[:, 2]


def _exact_lr(geo, nlayers, gate):
    x, y, z = _xyz(geo)
    t = np.asarray(geo.tn)
    LR = torch.zeros(x.numel(), x.numel(), dtype=torch.float64, device="cuda")
    for n1 in range(-3, 4):
        for n2 in range(-3, 4):
            if abs(n1 + n2) <= 3:
                s = n1 * t[:, 0] + n2 * t[:, 1]
                LR += _fv((x - s[0])[:, None], (y - s[1])[:, None], z[:, None], x[None], y[None], z[None], nlayers, gate)
    up = torch.triu(LR)
    return up + torch.triu(LR, 1).T


class _Exact:
    """One system in plain torch: tables, H(k), density matrix, energies (matrices indexed [i, j])."""

    def __init__(self, ntheta, nlayers, numk, nfilling, seed, long_range=True):
        S = _setup(ntheta, nlayers, numk, False, nfilling, "corrected")
        self.geo = geo = fg.build_geometry(S)
        self.n, self.nlayers, self.numk, self.nfilling = geo.Coords.shape[0], nlayers, numk, nfilling
        self.alpha = 5.853 / 10.0
        x, y, z = _xyz(geo)
        ri = (x[:, None], y[:, None], z[:, None])
        self.R = _cells(geo)
        self.tm, self.tp, self.vm, self.vp = [], [], [], []
        for R in self.R:
            for t, f, sign in ((self.tm, "t", -1), (self.tp, "t", 1), (self.vm, "v", -1), (self.vp, "v", 1)):
                rj = (x[None] + sign * R[0], y[None] + sign * R[1], z[None])
                t.append(_ft(*ri, *rj) if f == "t" else _fv(*ri, *rj, nlayers, XI))
        if long_range:
            self.LR = _exact_lr(geo, nlayers, XI)
        self.P = _field(geo, nfilling, seed).transpose(1, 2).contiguous()
        self.numb = min(20, self.n)
        self.nlow = (self.n - 2 * self.numb + 2 * (self.numb // 2)) // 2 + 1
        self.nup = (self.n + 2 * (self.numb // 2)) // 2

    def potential(self, dens):
        return 2 * self.alpha * (self.LR @ (dens - 0.5)) + HUBBARD_U * (dens - 0.5)

    def hamiltonian(self, k, V):
        """H(k) of momentum index k (0-based), the lower triangle mirrored."""
        i1, i2 = (int(v) for v in self.geo.nMomentaComponents[k])
        vk = self.geo.MomentaValues[i1, i2]
        H = self.tm[0] - self.alpha * self.vm[0] * self.P[0].conj() + torch.diag(V).to(torch.complex128)
        for c in range(1, 4):
            th = float(vk[0] * self.R[c][0] + vk[1] * self.R[c][1])
            e = complex(math.cos(th), -math.sin(th))
            H = H + (self.tm[c] - self.alpha * self.vm[c] * self.P[c].conj()) * e
            H = H + (self.tp[c] - self.alpha * self.vm[c].T * self.P[c].T) * e.conjugate()
        return torch.tril(H) + torch.tril(H, -1).mH

    def bloch(self, k):
        i1, i2 = (int(v) for v in self.geo.nMomentaComponents[k])
        a, b = np.asarray(self.geo.nUnitCell_1), np.asarray(self.geo.nUnitCell_2)
        return [complex(np.exp(-2j * math.pi * (i1 * a[c] + i2 * a[c] + i2 * b[c]) / self.numk)) for c in range(4)]

    def energies(self, P, dens):
        kin = (self.tm[0] * P[0].real).sum() + sum((self.tm[c] * P[c].real).sum() + (self.tp[c] * P[c].T.real).sum()
                                                   for c in range(1, 4))
        sq = [p.real ** 2 + p.imag ** 2 for p in P]
        fock = -0.5 * ((self.vm[0] * sq[0]).sum() + sum((self.vm[c] * sq[c]).sum() + (self.vp[c] * sq[c].T).sum()
                                                        for c in range(1, 4)))
        d = dens - 0.5
        return [float(kin), float(fock), float(2 * (d @ self.LR @ d)), float(d @ d)]

    def total(self, E):
        return 2 * self.alpha * E[1] + 2 * E[0] + HUBBARD_U * E[3] + self.alpha * E[2]

    def iteration(self, mixing, deg):
        n, nk = self.n, self.numk ** 2
        dens_in = self.P[0].diagonal().real.clone()
        V = self.potential(dens_in)
        E_in = self.energies(self.P, dens_in)
        bands = torch.empty(nk, self.numb, dtype=torch.float64, device="cuda")
        Pn = torch.zeros_like(self.P)
        window = []
        for k in range(nk):
            w, Z = torch.linalg.eigh(self.hamiltonian(k, V))
            bands[k] = w[self.nlow - 1:self.nup]
            window.append(Z[:, self.nlow - 1:self.nup].clone())
            C = Z[:, :self.nlow - 1].conj() @ Z[:, :self.nlow - 1].T
            for c, ph in enumerate(self.bloch(k)):
                Pn[c] += ph * C
        flat = bands.T.reshape(-1)   # index band * nk + k
        order = torch.argsort(flat, stable=True)
        e = flat[order].cpu().numpy()
        x = nk * (n // 2 - self.nlow + 1) + nk / 2.0 * self.nfilling
        nF = int(math.floor(x + 0.5)) if x >= 0 else -int(math.floor(-x + 0.5))
        ef = (e[nF - 1] + e[nF]) / 2.0
        full = int(np.sum(e - ef < -ENERGY_TOL))
        part = int(np.sum(np.abs(e - ef) < ENERGY_TOL))
        for q in range(full + part):
            band, k = divmod(int(order[q]), nk)
            wgt = 1.0
            if q >= full:
                d = (nF - full) / part
                wgt = complex(float(np.float32(d)), 8.0) if deg == "reference" else d
            psi = window[k][:, band]
            for c, ph in enumerate(self.bloch(k)):
                Pn[c] += (ph * wgt) * torch.outer(psi.conj(), psi)
        Pn /= nk
        dn = Pn[0].diagonal().real.clone()
        c0 = self.total(E_in)
        if mixing == "pulay":
            step, P = 1.0, self.P + 0.7 * (Pn - self.P)
        else:
            t1 = self.total(self.energies(Pn, dn))
            t2 = self.total(self.energies(0.5 * (self.P + Pn), 0.5 * (dens_in + dn)))
            c1 = 4 * t2 - t1 - 3 * c0
            c2 = t1 - c0 - c1
            step = -c1 / 2 / c2 if c2 > 0 and abs(-c1 / 2 / c2 - 0.5) < 0.5 else 1.0
            P = step * Pn + (1 - step) * self.P
        dens = P[0].diagonal().real.clone()
        E = self.energies(P, dens)
        Vn = self.potential(dens)
        ref = (Pn, self.potential(dn)) if mixing == "pulay" else (P, Vn)
        res = float((ref[1] - V).abs().max())
        for c in range(4):
            dP = (ref[0][c] - self.P[c]).abs()
            wf = self.vm[0].abs() if c == 0 else 0.5 * (self.vm[c] + self.vp[c].T).abs()
            res = max(res, float((self.alpha * wf * dP).max()))
        return {"energies": np.array(E), "total": np.array([c0, self.total(E)]), "fermi": np.array([ef]),
                "step": float(step), "residual": res, "density_change": float((dens - dens_in).abs().max()),
                "counts": np.array([nF, full + part, part, 0]),
                "P": P.transpose(1, 2).contiguous(), "density": dens, "potential": Vn}, bands


def exact(case, seed):
    kind = case["kind"]
    if kind == "scf":
        x = _Exact(case["ntheta"], case["nlayers"], case["numk"], case["nfilling"], seed)
        out, bands = x.iteration(case["mixing"], case["deg"])
        return dict(out, bands=bands.T.cpu().numpy())
    if kind == "bands":
        x = _Exact(case["ntheta"], case["nlayers"], case["numk"], case["nfilling"], seed)
        V = x.potential(x.P[0].diagonal().real)
        w = [torch.linalg.eigvalsh(x.hamiltonian(k, V))[x.nlow - 1:x.nup] for k in range(case["numk"] ** 2)]
        return {"bands": torch.stack(w, 1).cpu().numpy(), "info": 0}
    if kind == "group":
        return [_Exact(case[m], 2, case["numk"], case["nfilling"], seed + 7 * q).iteration("oda", case["deg"])[0]
                for q, m in enumerate(("m0", "m1", "m2"))]
    if kind == "zheevr":
        H = torch.tril(_matrix(case, seed))
        # the phases of eigenvectors are free: no exact value for them
        return {"info": 0, "w": torch.linalg.eigvalsh(H)[:case["iu"]], "Z": None}
    if kind == "mlp":
        p, x, y, shapes = _mlp_inputs(case, seed)
        p = torch.as_tensor(p).bfloat16().double()   # the network's weights are BF16
        parts = [q.reshape(s).requires_grad_(True) for q, s in zip(p.split([math.prod(s) for s in shapes]), shapes)]
        h = torch.as_tensor(x).double()
        for q in range(3):
            h = torch.nn.functional.silu(h @ parts[2 * q].T + parts[2 * q + 1])
        out = h @ parts[6].T + parts[7]
        loss = ((out - torch.as_tensor(y).double()) ** 2).sum() / x.shape[0]
        g = torch.autograd.grad(loss, parts)
        return {"rc": 0, "gradient": torch.cat([v.reshape(-1) for v in g]), "loss": float(loss.detach())}
    s = _gated(case, seed)
    return {"LR": _exact_lr(fg.build_geometry(s), case["nlayers"], s.xi).cpu().numpy()}
