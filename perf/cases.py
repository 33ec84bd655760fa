"""The band-structure work that users of this package have it do, as cases that can be timed.

A case names a material set, a plane-wave cutoff (shells), the terms of H(k) that are on (nonlocal
wells, spin-orbit), the precision of the solve, the number of bands and of k-points, and the entry
point ("call") that the work goes through:

  one       api.Hamiltonian: SetMatrix + Diagonalize of single k-points, as the direct users of the
            class loop over them (eigenvalues of the whole matrix)
  host      api.BandStructure.Compute_parallel on a k list: host k in, host energies out
  device    uepm_solve_device on device buffers (k, energies and status stay on the GPU)
  particles fbmc.BandQuery.energy_and_velocity_device: energies and velocities of Monte Carlo particles
  epsilon   dielectric.DielectricFunction.compute_dielectric_function: eigenvectors at k and k + q and
            their overlap sums over an energy grid
  batch     uepm_batch_run over the eight materials of serve.MIXED_SET, k-points dealt out unevenly

The k-points are seeded: uniform in the first Brillouin zone, as a zone integral or a Monte Carlo
ensemble has them, or ("path") on straight segments between zone points, as a band plot has them.
"""
from __future__ import annotations

import ctypes as C
import math
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import ultimateepm_gb300 as U
from ultimateepm_gb300 import _native as N
from ultimateepm_gb300.api import _Context
from ultimateepm_gb300.dielectric import FIRST_CONDUCTION_BAND, DielectricFunction
from ultimateepm_gb300.fbmc import BandQuery
from ultimateepm_gb300.serve import MIXED_SET

PARAMS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "params")
PREC = {"fp64": N.UEPM_PREC_FP64, "mixed": N.UEPM_PREC_MIXED}
CB, ALL, SID = "si-cohen-bergstresser.yaml", "materials.yaml", "si-nonlocal-d.yaml"


def _case(call, yaml, sym, shells, nl, soc, prec, bands, k, path=False, name=None):
    c = {"call": call, "yaml": yaml, "material": sym, "shells": shells, "nl": nl, "soc": soc, "precision": prec,
         "bands": bands, "k": k, "path": path}
    return dict({"name": name}, **c) if name else c


def listed():
    return [
        # a direct user of Hamiltonian: one k-point at a time, every eigenvalue (basis 137)
        _case("one", CB, "Si", 10, False, False, "fp64", 0, 1, name="one k, Si 137"),
        # a quick look at a band structure with the command line's default size: 60 points, host arrays
        _case("host", ALL, "GaAs", 12, True, False, "fp64", 30, 60, True, name="plot, GaAs 181, 60 k"),
        # the headline workload: 2000 points on a path, 16 bands, resident on the device
        _case("device", CB, "Si", 10, False, False, "mixed", 16, 2000, True, name="path, Si 137, mixed"),
        # the same through the drop-in class and in its precision
        _case("host", CB, "Si", 10, False, False, "fp64", 16, 2000, True, name="path, Si 137, fp64"),
        # zone sampling with nonlocal wells: real, complex and larger real matrices
        _case("device", SID, "Si", 10, True, False, "mixed", 12, 20000, name="zone, Si-d 137, mixed"),
        _case("host", ALL, "InP", 9, True, False, "mixed", 12, 20011, name="zone, InP 113, mixed"),
        _case("device", ALL, "Ge", 12, True, False, "mixed", 12, 10007, name="zone, Ge 181, mixed"),
        # zone sampling with spin-orbit coupling: the largest matrices
        _case("device", ALL, "Ge", 12, True, True, "mixed", 16, 3001, name="zone, Ge soc 362, mixed"),
        _case("device", ALL, "Ge", 12, True, True, "fp64", 16, 500, name="zone, Ge soc 362, fp64"),
        # a Monte Carlo ensemble's energies and velocities, in the class's default precision
        _case("particles", CB, "Si", 10, False, False, "fp64", 12, 16384, name="particles, Si 137, fp64"),
        # the dielectric function's sums at one q over 1001 energies
        _case("epsilon", CB, "Si", 10, False, False, "fp64", 16, 4096, name="epsilon, Si 137, fp64"),
        # eight materials, orders 89 to 458, four with spin-orbit, in one batch
        _case("batch", ALL, "*", 0, True, True, "mixed", 16, 6000, name="batch, 8 materials, mixed"),
    ]


def _order(c):
    return (2 if c["soc"] else 1) * len(U.generate_basis_vectors(c["shells"]))


def _flops(c):
    """The reduction to tridiagonal form of a matrix of this case, which the rest is small against."""
    real = not c["soc"] and c["material"] in ("Si", "Ge", "Sn")
    return (4.0 if real else 16.0) / 3.0 * _order(c) ** 3


def draw(rng):
    call = rng.choice(["one", "host", "host", "device", "device", "device", "particles", "epsilon", "batch"])
    if call == "batch":
        return _case("batch", ALL, "*", 0, True, True, "mixed", rng.randint(8, 16),
                     int(round(math.exp(rng.uniform(math.log(64), math.log(6000))))))
    if call in ("particles", "epsilon"):
        yaml, sym, nl, soc, prec = CB, "Si", False, False, "fp64"
        shells = rng.randint(6, 11)
    else:
        yaml, sym = rng.choice([(CB, "Si"), (SID, "Si")] + [(ALL, m) for m, _, _ in MIXED_SET] * 2)
        nl = yaml != CB and sym != "AlAs" and rng.random() < 0.75
        soc = yaml == ALL and sym in ("Si", "Ge", "GaAs", "GaP") and rng.random() < 0.5
        prec = "fp64" if call == "one" else rng.choice(["fp64", "mixed", "mixed"])
        shells = rng.randint(8, 13)
    c = _case(call, yaml, sym, shells, nl, soc, prec, rng.randint(8, 16) if call != "one" else 0, 1,
              call in ("host", "device") and rng.random() < 0.5)
    most = 20000 if call != "one" else 8
    most = min(most, int((2.5e10 if call == "epsilon" else 5e10 if prec == "fp64" else 5e11) / _flops(c)))
    least = {"one": 1, "host": 20, "device": 100, "particles": 100, "epsilon": 100}[call]
    c["k"] = int(round(math.exp(rng.uniform(math.log(least), math.log(max(most, least + 1))))))
    return c


# ---- inputs ---------------------------------------------------------------------------------------

def _zone(n, rng):
    """Uniform in the first zone (|k_i| <= 1, |kx| + |ky| + |kz| <= 3/2), units of 2 pi / a."""
    out = np.empty((0, 3))
    while len(out) < n:
        c = rng.uniform(-1.0, 1.0, size=(2 * (n - len(out)) + 8, 3))
        out = np.concatenate([out, c[np.abs(c).sum(axis=1) <= 1.5]])
    return np.ascontiguousarray(out[:n])


def _kpoints(c, rng):
    if not c["path"]:
        return _zone(c["k"], rng)
    p = _zone(10, rng)  # nine segments
    t = np.linspace(0.0, 9.0, c["k"], endpoint=False)
    i = t.astype(int)
    return np.ascontiguousarray(p[i] + (t - i)[:, None] * (p[i + 1] - p[i]))


def _materials(yaml):
    m = U.Materials()
    m.load_material_parameters(os.path.join(PARAMS, yaml))
    return m.materials


def _groups(c, rng):
    """The batch's groups that get k-points: (symbol, shells, spin-orbit, k); how many each, the case says."""
    share = np.random.default_rng(c["k"])
    counts = share.multinomial(c["k"], share.dirichlet(np.full(len(MIXED_SET), 4.0)))
    return [(sym, sh, so, _zone(int(n), rng)) for (sym, sh, so), n in zip(MIXED_SET, counts) if n]


def _inputs(c, seed):
    """Everything that the seed gives, as numpy arrays."""
    rng = np.random.default_rng(seed)
    if c["call"] == "batch":
        return {"groups": _groups(c, rng)}
    d = {"k": _kpoints(c, rng)}
    if c["call"] == "particles":
        d["band"] = rng.integers(4, c["bands"], size=c["k"])
        d["band"][0] = c["bands"] - 1
    if c["call"] == "epsilon":
        d["q"] = rng.uniform(0.05, 0.4, size=3)
    return d


def _eps_energies():
    return np.linspace(0.0, 20.0, 1001)


def _ptr(t):
    return C.c_void_p(t.data_ptr())


class _Batch:
    """A uepm_batch and the buffers and contexts that it runs on."""

    def __init__(self, c, groups):
        L, mats = N.load(), _materials(c["yaml"])
        self.b, self.ctx, self.bufs = C.c_void_p(), [], []
        N.check(L.uepm_batch_create(C.byref(self.b)))
        for sym, sh, so, k in groups:
            m = mats[sym]
            x = _Context(m, U.generate_basis_vectors(sh), bool(m.raw.has_nonlocal), so, PREC[c["precision"]])
            t = (torch.from_numpy(k).cuda(), torch.zeros((len(k), c["bands"]), dtype=torch.float64, device="cuda"),
                 torch.zeros(len(k), dtype=torch.int32, device="cuda"))
            N.check(L.uepm_batch_add(self.b, x.h, _ptr(t[0]), len(k), c["bands"], N.UEPM_WANT_VALUES, _ptr(t[1]), None,
                                     None, _ptr(t[2])))
            self.ctx.append(x)
            self.bufs.append(t)

    def run(self):
        N.check(N.load().uepm_batch_run(self.b, C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return [t[1:] for t in self.bufs]

    def __del__(self):
        torch.cuda.synchronize()
        N.load().uepm_batch_destroy(self.b)
        for x in self.ctx:
            x.close()


def prepare(case, seed):
    c, d = case, _inputs(case, seed)
    s = {"case": c}
    if c["call"] == "batch":
        s["batch"] = _Batch(c, d["groups"])
        return s
    m = _materials(c["yaml"])[c["material"]]
    if c["call"] == "one":
        s["k"], s["h"] = d["k"], U.Hamiltonian(m, U.generate_basis_vectors(c["shells"]))
    elif c["call"] == "host":
        s["bs"] = U.BandStructure()
        s["bs"].set_precision(c["precision"])
        s["bs"].Initialize(m, c["bands"] // 2 if c["soc"] else c["bands"], d["k"], c["shells"], c["nl"], c["soc"])
    elif c["call"] == "device":
        s["ctx"] = _Context(m, U.generate_basis_vectors(c["shells"]), c["nl"], c["soc"], PREC[c["precision"]])
        s["k"] = torch.from_numpy(d["k"]).cuda()
        s["E"] = torch.zeros((c["k"], c["bands"]), dtype=torch.float64, device="cuda")
        s["st"] = torch.zeros(c["k"], dtype=torch.int32, device="cuda")
    elif c["call"] == "particles":
        s["q"] = BandQuery(m, c["shells"])
        s["k"] = torch.from_numpy(d["k"] / s["q"].scale).cuda()
        s["band"] = torch.from_numpy(d["band"]).cuda()
    else:
        f = DielectricFunction(m, U.generate_basis_vectors(c["shells"]), c["bands"])
        f.m_kpoints = d["k"]
        f.set_nb_kpoints(c["k"])
        f.set_energies(_eps_energies())
        f.set_qpoints([d["q"]])
        s["f"] = f
    return s


def run(s):
    c = s["case"]
    if c["call"] == "one":
        out = []
        for k in s["k"]:
            s["h"].SetMatrix(k, c["nl"], c["soc"])
            s["h"].Diagonalize(False)
            out.append(s["h"].eigenvalues())
        return out
    if c["call"] == "host":
        s["bs"].Compute_parallel()
        return s["bs"].get_band_energies()
    if c["call"] == "device":
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        N.check(N.load().uepm_solve_device(s["ctx"].h, _ptr(s["k"]), c["k"], c["bands"], N.UEPM_WANT_VALUES, _ptr(s["E"]),
                                           None, None, _ptr(s["st"]), st))
        return s["E"], s["st"]
    if c["call"] == "particles":
        return s["q"].energy_and_velocity_device(s["k"], s["band"])
    if c["call"] == "epsilon":
        f = s["f"]
        f.m_dielectric_function_real = []
        f.compute_dielectric_function()
        return f.get_flat_dielectric_function()
    return s["batch"].run()


def work(case):
    c = case
    if c["call"] == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for sym, sh, so in MIXED_SET:
            w = work(_case("device", ALL, sym, sh, True, so, "mixed", c["bands"], c["k"] / len(MIXED_SET)))
            total = {q: total[q] + w[q] for q in total}
        return total
    nb = {"one": _order(c), "host": c["bands"] // 2 * 2 if c["soc"] else c["bands"]}.get(c["call"], c["bands"])
    n_solves = 2 * c["k"] if c["call"] == "epsilon" else c["k"]
    out = {"particles": 32 * c["k"], "epsilon": 8 * 1001}.get(c["call"], 8 * nb * c["k"])
    return {"bytes": 24.0 * c["k"] + out, "flops": _flops(c) * n_solves}


# ---- the same values in plain 64-bit torch --------------------------------------------------------

PLANCK, Q_E, M_E, BOHR = 6.62607015e-34, 1.602176634e-19, 9.1093837015e-31, 5.29177210903e-11
HBAR = PLANCK / (2.0 * math.pi)


def _j(l, x):
    """Spherical Bessel j_l, l = -1 .. 3: closed forms, and the power series where these cancel."""
    if l == -1:
        return torch.cos(x) / x
    y = x.clamp(min=0.5)
    s, co = torch.sin(y), torch.cos(y)
    far = {0: lambda: s / y, 1: lambda: s / y ** 2 - co / y, 2: lambda: (3 / y ** 3 - 1 / y) * s - 3 / y ** 2 * co,
           3: lambda: (15 / y ** 4 - 6 / y ** 2) * s - (15 / y ** 3 - 1 / y) * co}[l]()
    z, t = x.clamp(max=0.5), torch.ones_like(x)
    near = torch.ones_like(x)
    for i in range(1, 12):
        t = t * (-0.5 * z * z) / (i * (2 * l + 2 * i + 1))
        near = near + t
    near = near * z ** l / math.prod(range(1, 2 * l + 2, 2))
    return torch.where(x < 0.5, near, far)


def _i2(x):
    y = x.clamp(min=1.0)
    far = ((y * y + 3) * torch.sinh(y) - 3 * y * torch.cosh(y)) / y ** 3
    z, t = x.clamp(max=1.0), torch.ones_like(x)
    near = torch.ones_like(x)
    for i in range(1, 14):
        t = t * (0.5 * z * z) / (i * (2 * i + 5))
        near = near + t
    return torch.where(x < 1.0, near * z * z / 15.0, far)


def _well(n1, n2, R, l):
    """The square well's F_l of |K1| and |K2| (1/m)."""
    far = R ** 2 / (n1 * n1 - n2 * n2) * (n1 * _j(l + 1, n1 * R) * _j(l, n2 * R) - n2 * _j(l + 1, n2 * R) * _j(l, n1 * R))
    same = R ** 3 / 2.0 * (_j(l, n1 * R) ** 2 - _j(l - 1, n1 * R) * _j(l + 1, n1 * R))
    return torch.where((n1 - n2).abs() > 1e-4, far, same)


def _matrix(p, shells, nl, soc, k):
    """H(k) [c, n, n] (eV) of the material parameters p."""
    dev, f8 = k.device, torch.float64
    G = torch.as_tensor(U.generate_basis_vectors(shells), device=dev, dtype=f8)
    a = 1e-10 * p.lattice_constant
    ff, vol = 2 * math.pi / a, a ** 3 / 8
    df = HBAR ** 2 / (2 * M_E * Q_E)
    D = G[:, None] - G[None, :]
    d2, ph = (D * D).sum(-1).round(), D.sum(-1) * (math.pi / 4)
    VS = sum(v * (d2 == g).to(f8) for g, v in ((3, p.V3S), (4, p.V4S), (8, p.V8S), (11, p.V11S)))
    VA = sum(v * (d2 == g).to(f8) for g, v in ((3, p.V3A), (4, p.V4A), (8, p.V8A), (11, p.V11A)))
    H = torch.complex(VS * torch.cos(ph), VA * torch.sin(ph)).expand(len(k), -1, -1).clone()
    K = k[:, None] + G[None]
    H.diagonal(dim1=1, dim2=2).add_(ff * ff * df * (K * K).sum(-1))
    if nl:
        n = ff * K.norm(dim=-1)
        n1, n2 = n[:, :, None].expand(H.shape), n[:, None, :].expand(H.shape)
        cosang = (ff * ff * (K[:, :, None] * K[:, None, :]).sum(-1) / (n1 * n2)).nan_to_num(1.0)
        kF2 = (96 * math.pi ** 2) ** (2.0 / 3.0) / a ** 2

        def atom(al, be, A2, R0, R2):
            v = torch.zeros(H.shape, device=dev, dtype=f8)
            if R0:
                v = v + 4 * math.pi / vol * (al + df * be * (n1 * n2 - kF2)) * _well(n1, n2, R0, 0)
            if A2:
                P2 = 0.5 * (3 * cosang ** 2 - 1)
                if p.nl_well == 1:
                    v = v + 20 * math.pi / vol * A2 * P2 * _well(n1, n2, R2, 2)
                else:
                    g = _i2(0.5 * R2 * R2 * n1 * n2) * torch.exp(-0.25 * (n1 * n1 + n2 * n2) * R2 * R2)
                    v = v + 5 * math.pi ** 1.5 * R2 ** 3 / vol * A2 * P2 * g
            return v

        va = atom(p.alpha0_anion, p.beta0_anion, p.A2_anion, p.R0_anion, p.R2_anion)
        vc = atom(p.alpha0_cation, p.beta0_cation, p.A2_cation, p.R0_cation, p.R2_cation)
        H = H + torch.complex(torch.cos(ph) * (va + vc) / 2, torch.sin(ph) * (va - vc) / 2)
    if not soc:
        return H

    def B(period, r):
        q = (ff * K.norm(dim=-1) * BOHR / r) ** 2
        return {2: 1 / (1 + q) ** 3, 3: (5 - q) / (5 * (1 + q) ** 4), 4: (5 - 3 * q) / (5 * (1 + q) ** 5)}[period]

    bc, ba = B(p.period_cation, p.radial_extent_cation), B(p.period_anion, p.radial_extent_anion)
    l1, l2 = p.mu_soc * bc[:, :, None] * bc[:, None, :], p.alpha_soc * p.mu_soc * ba[:, :, None] * ba[:, None, :]
    phase = torch.complex((l1 - l2) / 2 * torch.sin(ph), -(l1 + l2) / 2 * torch.cos(ph))
    X = torch.linalg.cross(K[:, :, None].expand(-1, -1, len(G), -1), K[:, None].expand(-1, len(G), -1, -1))
    cx, cy, cz = X[..., 0], -X[..., 1], X[..., 2]  # the y component as the reference writes it
    top = torch.cat([H + cz * phase, torch.complex(cx, cy) * phase], dim=2)
    low = torch.cat([torch.complex(cx, -cy) * phase, H - cz * phase], dim=2)
    return torch.cat([top, low], dim=1)


def _states(p, c, k, vectors=False, nb=None):
    """Eigenvalues [k, nb] and, if asked, eigenvectors [k, n, nb]: LAPACK on the host's cores, on the GPU afterwards."""
    def solve(H):
        torch.set_num_threads(1)  # per thread: the pool's threads each solve matrices of their own
        return torch.linalg.eigh(H) if vectors else (torch.linalg.eigvalsh(H), None)

    E, X = [], []
    with ThreadPoolExecutor(len(os.sched_getaffinity(0))) as pool:
        for part in torch.as_tensor(k).cuda().split(512):
            H = _matrix(p, c["shells"], c["nl"], c["soc"], part)
            H = (H if H.imag.any() else H.real.contiguous()).cpu()
            for e, x in pool.map(solve, H.split(8)):
                E.append(e[:, :nb])
                X.append(x[:, :, :nb] if vectors else None)
    return torch.cat(E).cuda(), torch.cat(X).cuda() if vectors else None


def exact(case, seed):
    c, d = case, _inputs(case, seed)
    mats = _materials(c["yaml"])
    if c["call"] == "batch":
        out = []
        for sym, sh, so, k in d["groups"]:
            g = dict(c, material=sym, shells=sh, soc=so, nl=bool(mats[sym].raw.has_nonlocal))
            out.append((_states(mats[sym].raw, g, k, nb=c["bands"])[0], None))
        return out
    p = mats[c["material"]].raw
    if c["call"] == "one":
        return [x.cpu().numpy() for x in _states(p, c, d["k"])[0]]
    if c["call"] == "host":
        return _states(p, c, d["k"], nb=c["bands"] // 2 * 2 if c["soc"] else c["bands"])[0].cpu().numpy()
    if c["call"] == "device":
        return _states(p, c, d["k"], nb=c["bands"])[0], None
    a, df = 1e-10 * p.lattice_constant, HBAR ** 2 / (2 * M_E * Q_E)
    E, X = _states(p, c, d["k"], True, c["bands"])
    if c["call"] == "particles":
        rows, b = torch.arange(c["k"], device="cuda"), torch.as_tensor(d["band"]).cuda()
        G = torch.as_tensor(U.generate_basis_vectors(c["shells"]), device="cuda", dtype=torch.float64)
        w = X.abs().square()[rows, :, b]
        # dE/dk (eV m) of the kinetic term, over h_bar in eV s
        g = 2 * df * (2 * math.pi / a) * (torch.as_tensor(d["k"]).cuda() * w.sum(1)[:, None] + w @ G)
        return E[rows, b], g * Q_E / HBAR
    E2, X2 = _states(p, c, d["k"] + d["q"], True, c["bands"])
    fc, w, eta2 = FIRST_CONDUCTION_BAND, torch.as_tensor(_eps_energies()).cuda(), 1e-4
    O = (X2[:, :, fc:].transpose(1, 2) @ X[:, :, :fc]).abs().square()
    dE = E2[:, fc:, None] - E[:, None, :fc]
    total = torch.zeros_like(w)
    for o, e in zip(O.reshape(-1).split(1 << 15), dE.reshape(-1).split(1 << 15)):
        lo, hi = e[:, None] - w, e[:, None] + w
        total += o @ (lo / (lo * lo + eta2) + hi / (hi * hi + eta2))
    return total.cpu().numpy()
