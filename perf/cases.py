"""The measured cases: what users of the lattice library have it do between two outputs of a run.

A run advances its lattice by an output interval and reads the result: the volume averages and the
state (a snapshot, in pinned host memory).  Each case is such an interval of one model, through
Lattice / LatticeBatch and, for reads into memory that the program keeps, the C ABI that they bind.
The sizes are those of the benchmark's workloads and of the tests, with odd lattices beside them.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from cosmolattice_b200 import MODELS, Lattice, ParameterParser, RunParameters, _capi
from cosmolattice_b200.batch import LatticeBatch

F_STAR = 5.6964e18      # homogeneous field of the singlet and U(1) runs, GeV
F_STAR_D = 5.25151e18   # homogeneous doublet of the SU(2) x U(1) runs, GeV
M_PL = 2.435e18         # reduced Planck mass, GeV
G_U1, G_U1_SU2, G_SU2 = 0.5, 0.35, 0.6
Q_SINGLET, Q_GH = 1.5, 50.0
AMP = 1e-3              # rms of the fluctuations
W4 = 1.351207191959657771818, -1.702414403875838200264  # fourth-order Verlet weights: W4[0], W4[1], W4[0]
GAUGE_FRACTION = (0.0, 0.0, 1.0, 1.0, 0.0)
GAUGE_FRACTION_SU2 = (0.0,) * 6 + (1.0, 1.0, 1.0, 1.0, 0.0)
COMPS = {"singlet": (1, 1), "gws": (1, 1), "u1": (5, 5), "u1_gradient": (5, 5), "su2": (22, 19), "su2_tangent": (22, 19)}


def listed():
    def case(name, kind, N, steps, evolver="VV2", precision="fp64", fields=1, **more):
        return dict(name=name, kind=kind, N=N, steps=steps, evolver=evolver, precision=precision, fields=fields, **more)

    return [
        # the 64^3 run with the default frequent output (every ten steps): launches and latency
        case("singlet_64", "singlet", 64, 10),
        # the two-field header of the reference with its default evolver, on a ragged lattice
        case("singlet2_125_lf", "singlet", 125, 100, evolver="LF", fields=2),
        # a production lattice in the FP32 storage form
        case("singlet_384_fp32", "singlet", 384, 200, precision="fp32"),
        # the headline lattice
        case("singlet_512", "singlet", 512, 200),
        # gravitational waves beside the scalar, with the spectra of both at the output
        case("gws_128", "gws", 128, 50),
        # charged scalar and U(1) field, fourth order
        case("u1_128_vv4", "u1", 128, 50, evolver="VV4"),
        # the same model, leapfrog, FP32 storage, odd lattice
        case("u1_99_lf_fp32", "u1", 99, 100, evolver="LF", precision="fp32"),
        # one gradient of the final gauge-energy fraction: an iteration of a parameter fit
        case("u1_gradient_96", "u1_gradient", 96, 40, evolver="VV4", every=10),
        # SU(2) x U(1) with scalar, charged scalar and doublet
        case("su2_192", "su2", 192, 30),
        # the same in the FP32 storage form on an odd lattice
        case("su2_95_fp32", "su2", 95, 60, precision="fp32"),
        # its derivative along g_SU2, advanced beside the state
        case("su2_tangent_80", "su2_tangent", 80, 20),
        # many small lattices of different sizes in one batch
        case("ensemble_48_fp32", "ensemble", 96, 100, precision="fp32", members=48),
    ]


def draw(rng):
    kind = rng.choice(["singlet"] * 4 + ["u1", "u1", "su2", "su2", "gws", "u1_gradient", "su2_tangent", "ensemble"])
    lo, hi = {"singlet": (32, 400), "gws": (32, 160), "u1": (32, 160), "u1_gradient": (24, 96), "su2": (24, 160),
              "su2_tangent": (24, 80), "ensemble": (48, 96)}[kind]
    N = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    precision = rng.choice(["fp64", "fp32"])
    evolver = rng.choice(["LF", "VV2", "VV4"])
    steps = int(round(math.exp(rng.uniform(math.log(10), math.log(60)))))
    c = dict(kind=kind, N=N, steps=steps, evolver=evolver, precision=precision, fields=1)
    if kind == "singlet":
        c["fields"] = rng.choice([1, 2])
    elif kind == "u1_gradient":
        c.update(every=rng.choice([5, 8, 10]), steps=rng.randint(10, 40))
    elif kind == "su2_tangent":
        c["steps"] = rng.randint(5, 20)
    elif kind == "ensemble":
        c.update(N=N - N % 4, members=rng.randint(6, 48), evolver=rng.choice(["VV2", "VV4"]))
    return c


# ---- inputs --------------------------------------------------------------------------------------
def _member_sizes(case):
    """Lattice sizes of an ensemble: its largest, and two thirds, a half and a third of it, in turn."""
    N = case["N"]
    return [max(16, int(N * (1, 2 / 3, 1 / 2, 1 / 3)[i % 4]) // 4 * 4) for i in range(case["members"])]


def _dx(case, N):
    # the benchmark's spacings: that of the 64^3 box (2 pi / 64) for the singlets at every size,
    # a box of side 2 pi for the gauge models
    return 2 * math.pi / (64 if case["kind"] in ("singlet", "gws") else N)


def _dt(case):
    return 0.01 if case["kind"] in ("singlet", "gws", "ensemble") else 0.005


class _Noise:
    """Smooth random fields of unit rms: white noise cut off at a quarter of the lattice's modes and
    weighted as vacuum fluctuations are."""

    def __init__(self, N, seed):
        self.N, self.gen = N, torch.Generator("cuda").manual_seed(seed)
        k = torch.fft.fftfreq(N, 1 / N, device="cuda", dtype=torch.float64)
        kz = torch.fft.rfftfreq(N, 1 / N, device="cuda", dtype=torch.float64)
        k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
        self.filt = torch.where(k2 <= (N / 4) ** 2, (k2 + 1) ** -0.25, 0.0)
        self.filt[0, 0, 0] = 0.0

    def __call__(self, rms=AMP):
        n = torch.randn((self.N,) * 3, generator=self.gen, device="cuda", dtype=torch.float64)
        n = torch.fft.irfftn(torch.fft.rfftn(n) * self.filt, s=n.shape)
        return n * (rms / n.square().mean().sqrt())


def _qexp(v):
    """exp(i v . sigma) as the quaternion (cos |v|, sin |v| v / |v|); v: three fields."""
    n = (v[0] ** 2 + v[1] ** 2 + v[2] ** 2).sqrt()
    s = torch.sin(n) / n
    return [torch.cos(n), s * v[0], s * v[1], s * v[2]]


def _start(case, N, seed):
    """Fields and momenta of one lattice, on the GPU."""
    kind, noise = case["kind"], _Noise(N, seed)
    if kind in ("singlet", "gws", "ensemble"):
        nf = case["fields"]
        f = [noise() + (1.0 if i == 0 else 0.0) for i in range(nf)]
        p = [noise(4 * AMP) for i in range(nf)]
    elif kind in ("u1", "u1_gradient"):
        f = [noise() + math.sqrt(0.5) for _ in range(2)] + [noise() for _ in range(3)]
        p = [noise(4 * AMP) for _ in range(2)] + [noise() for _ in range(3)]
    else:
        f = [noise(), noise(), noise()] + [noise() + 0.5 for _ in range(4)] + [noise() for _ in range(3)]
        for _ in range(3):
            f += _qexp([noise() for _ in range(3)])
        p = [noise(4 * AMP) for _ in range(7)] + [noise() for _ in range(12)]
    return torch.stack(f), torch.stack(p)


def _model(case, N):
    kind = case["kind"]
    par = {"N": N, "dx": repr(_dx(case, N)), "dt": _dt(case), "evolver": case["evolver"], "expansion": "true", "lambda": 1.0}
    if kind in ("u1", "u1_gradient"):
        name = "lphi4U1"
        par.update(cmplx_field_initial_norm=F_STAR, gU1s=G_U1)
    elif kind in ("su2", "su2_tangent"):
        name = "lphi4SU2U1"
        par.update(qG=Q_GH, qH=Q_GH, SU2Doublet_initial_norm=F_STAR_D, gU1s=G_U1_SU2, gSU2s=G_SU2)
    elif case["fields"] == 2:
        name = "lphi4"
        par.update(initial_amplitudes=f"{F_STAR} 0", q=Q_SINGLET)
    else:
        name = "lphi4_1f"
        par.update(initial_amplitudes=F_STAR)
    par = ParameterParser(params=par)
    rp = RunParameters(par)
    return MODELS[name](par, rp), rp


SF = {"aI": 1.0, "aSI": 1.0, "aIM": 1.0, "aDotI": 0.0, "aDotSI": 0.0}


def _pinned(x):
    return torch.empty(x.shape, dtype=torch.float64, pin_memory=True).copy_(x)


def _ptr(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_double))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        sizes = _member_sizes(case)
        lat = LatticeBatch([_model(case, N) for N in sizes], precision=case["precision"])
        offs = np.concatenate([[0], np.cumsum([N ** 3 for N in sizes])])
        out = torch.empty((2, int(offs[-1])), dtype=torch.float64, pin_memory=True)
        for i, N in enumerate(sizes):
            f, p = _start(case, N, 1000 * seed + i)
            out[0, offs[i]:offs[i + 1]] = f.flatten()
            out[1, offs[i]:offs[i + 1]] = p.flatten()
            lat.set_state(i, out[0, offs[i]:offs[i + 1]].numpy(), out[1, offs[i]:offs[i + 1]].numpy(), SF)
        lat.initialize()
        return {"case": case, "lat": lat, "out": out, "offs": offs}
    f, p = _start(case, case["N"], seed)
    model, rp = _model(case, case["N"])
    lat = Lattice(model, rp, precision=case["precision"])
    s = {"case": case, "lat": lat, "f": _pinned(f), "p": _pinned(p)}
    if kind == "gws":
        lat.gws_enable()
        s["gw"] = [torch.empty((5, *f.shape[1:]), dtype=torch.float64, pin_memory=True) for _ in range(2)]
    if kind == "u1_gradient":  # every pass starts from the same state and returns its gradient
        s["fbar"], s["pbar"] = _pinned(f), _pinned(p)
        s["weights"] = np.array(GAUGE_FRACTION)
        return s
    lat.set_state(s["f"].numpy(), s["p"].numpy(), SF)
    if kind == "su2_tangent":
        dp = np.zeros(s["p"].shape)
        dp[10:] = -s["p"].numpy()[10:] / G_SU2
        lat.tangent_begin([0, 0, 0, 0, 1.0, 0], momenta_dot=dp)
        s["df"], s["dp"] = (torch.empty_like(s[k], pin_memory=True) for k in "fp")
    lat.initialize()
    return s


# ---- one pass ------------------------------------------------------------------------------------
def _run_ensemble(s):
    lat, out, offs = s["lat"], s["out"], s["offs"]
    lat.evolve(s["case"]["steps"])
    sf, a = _capi.ScaleFactor(), []
    for i in range(len(offs) - 1):
        lat._check(lat.lib.clb_batch_get_state(lat.h, i, _ptr(out[0, offs[i]:]), _ptr(out[1, offs[i]:]), C.byref(sf)))
        a.append((sf.aI, sf.aDotI))
    return {"fields": out[0], "momenta": out[1], "a": np.array(a)}


def _run_gradient(s):
    lat, c = s["lat"], s["case"]
    lat.set_state(s["f"].numpy(), s["p"].numpy(), SF)
    lat.initialize()
    obs = lat.forward(c["steps"], c["every"], s["weights"])
    g = _capi.AdjointGrad()
    lat._check(lat.lib.clb_backward(lat.h, 1, _ptr(s["fbar"]), _ptr(s["pbar"]), C.byref(g)))
    return {"observable": np.array([obs]), "fields_bar": s["fbar"], "momenta_bar": s["pbar"],
            "couplings": np.array([g.dO_dcouplings[0], g.dO_dcouplings[1]])}


def run(s):
    kind = s["case"]["kind"]
    if kind == "ensemble":
        return _run_ensemble(s)
    if kind == "u1_gradient":
        return _run_gradient(s)
    lat, sf = s["lat"], _capi.ScaleFactor()
    lat.evolve(s["case"]["steps"])
    lat.sync()
    out = {"fields": s["f"], "momenta": s["p"]}
    if kind == "su2_tangent":
        out["observable"] = np.array(lat.tangent_observable(GAUGE_FRACTION_SU2))
        lat._check(lat.lib.clb_tangent_get_state(lat.h, _ptr(s["df"]), _ptr(s["dp"]), C.byref(sf)))
        out.update(fields_dot=s["df"], momenta_dot=s["dp"])
    else:
        out["energies"] = np.array(lat.measure()["energies"])
    if kind == "gws":
        out["spectra"] = np.stack([lat.spectrum(which=w)[1] for w in (0, 1)] + [lat.gw_spectrum()[1]])
        lat._check(lat.lib.clb_gws_get_state(lat.h, *map(_ptr, s["gw"])))
        out["gw"] = s["gw"]
    lat._check(lat.lib.clb_get_state(lat.h, _ptr(s["f"]), _ptr(s["p"]), C.byref(sf)))
    out["a"] = np.array([sf.aI, sf.aDotI])
    return out


def work(case):
    """Each stage reads and writes the state once, and the snapshot is written once; operations per
    site and stage as the model's kernels and drifts have them."""
    kind, esz = case["kind"], 8 if case["precision"] == "fp64" else 4
    stages = case["steps"] * (3 if case["evolver"] == "VV4" else 1)
    if kind == "ensemble":
        sites, comps, flops = sum(N ** 3 for N in _member_sizes(case)), 2, 30
    else:
        nf, npm = COMPS[kind]
        if kind in ("singlet", "gws"):
            nf = npm = case["fields"]
        sites, comps = case["N"] ** 3, nf + npm
        flops = {"singlet": 30 * nf, "gws": 30, "u1": 450, "u1_gradient": 2200, "su2": 2200, "su2_tangent": 6000}[kind]
    moved = {"u1_gradient": 4, "su2_tangent": 2}.get(kind, 1)  # the adjoint's recompute and sweep; the tangent
    b = 2.0 * comps * esz * moved * sites * stages + 8.0 * comps * moved * sites
    f = float(flops) * sites * stages
    if kind == "gws":  # ten more arrays, advanced once a step
        b, f = b + 20.0 * esz * sites * case["steps"] + 80.0 * sites, f + 100.0 * sites * case["steps"]
    return {"bytes": b, "flops": f}


# ---- the same in plain torch, FP64 ---------------------------------------------------------------
def _up(f, d):
    return torch.roll(f, -1, d - 3)


def _dn(f, d):
    return torch.roll(f, 1, d - 3)


def _mean(f):
    return f.mean((-3, -2, -1))


def _lapl(f, dx):
    s = -6 * f
    for d in range(3):
        s = s + _up(f, d) + _dn(f, d)
    return s / dx ** 2


def _cell(a):
    """A per-lattice number (or one per lattice of a stack) against its sites."""
    return a[..., None, None, None] if torch.is_tensor(a) else a


def _abs2(z):
    return z.real ** 2 + z.imag ** 2


class _Singlet:
    def __init__(self, case, N):
        self.dx, self.ns = _dx(case, N), case["fields"]
        self.fm2 = (F_STAR / M_PL) ** 2

    def kernel(self, f, a):
        a = _cell(a)
        out = []
        for i in range(self.ns):
            dv = f[i] ** 3 if i == 0 else Q_SINGLET * f[1] * f[0] ** 2
            if i == 0 and self.ns == 2:
                dv = dv + Q_SINGLET * f[0] * f[1] ** 2
            out.append(a ** 2 * _lapl(f[i], self.dx) - a ** 4 * dv)
        return out

    def drift(self, f, p, aS, h):
        return [x + _cell(h * aS ** -2) * y for x, y in zip(f, p)]

    def momenta(self, p):
        return [_mean(x ** 2) for x in p]

    def fields(self, f):
        g = [sum(_mean((_up(x, d) - x) ** 2) for d in range(3)) / self.dx ** 2 for x in f]
        v = [0.25 * _mean(f[0] ** 4)] + ([0.5 * Q_SINGLET * _mean((f[0] * f[1]) ** 2)] if self.ns == 2 else [])
        return g, v

    def energies(self, pi2, fl, a):
        """[(kind, value)]: kinetic, gradient, gauge or potential."""
        out = []
        for i in range(self.ns):
            out += [("K", 0.5 * pi2[i] * a ** -6), ("G", 0.5 * fl[0][i] * a ** -2)]
        return out + [("V", v) for v in fl[1]]


class _U1:
    def __init__(self, case, N, c4=1.0, g=G_U1):
        self.dx, self.fm2, self.c4, self.g = _dx(case, N), (F_STAR / M_PL) ** 2, c4, g

    def links(self, A, g):
        return [torch.exp(-1j * self.dx * g * A[i]) for i in range(3)]

    def curl(self, A):
        out = []
        for i in range(3):
            grad = 0
            for j in range(3):
                t = (_up(A[j], i) - A[j]) / self.dx
                grad = grad + (t - _dn(t, j)) / self.dx
            out.append(_lapl(A[i], self.dx) - grad)
        return out

    def b2(self, A):
        F = lambda i, j: (_up(A[j], i) - A[j] - _up(A[i], j) + A[i]) / self.dx  # noqa: E731
        return _mean(F(1, 0) ** 2 + F(2, 0) ** 2 + F(2, 1) ** 2)

    def kernel(self, f, a):
        phi, A = torch.complex(f[0], f[1]), f[2:]
        U = self.links(A, self.g)
        fw = [U[d] * _up(phi, d) for d in range(3)]
        lap = sum(fw[d] + _dn(U[d].conj() * phi, d) for d in range(3)) - 6 * phi
        k = a ** 2 * lap / self.dx ** 2 - a ** 4 / 2 * 4 * self.c4 * _abs2(phi) * phi
        curl = self.curl(A)
        J = [2 / self.dx * self.g * (fw[i].conj() * phi).imag for i in range(3)]
        return [k.real, k.imag] + [curl[i] - a ** 2 * J[i] for i in range(3)]

    def drift(self, f, p, aS, h):
        return [x + h * aS ** -2 * y for x, y in zip(f[:2], p[:2])] + [x + h * y for x, y in zip(f[2:], p[2:])]

    def momenta(self, p):
        return [_mean(p[0] ** 2 + p[1] ** 2), _mean(p[2] ** 2 + p[3] ** 2 + p[4] ** 2)]

    def fields(self, f):
        phi = torch.complex(f[0], f[1])
        U = self.links(f[2:], self.g)
        g = sum(_mean(_abs2(U[d] * _up(phi, d) - phi)) for d in range(3)) / self.dx ** 2
        return [g, self.b2(f[2:])], [self.c4 * _mean(_abs2(phi) ** 2)]

    def energies(self, pi2, fl, a):
        return [("K", pi2[0] * a ** -6), ("G", fl[0][0] * a ** -2), ("E", 0.5 * a ** -4 * pi2[1]),
                ("E", 0.5 * a ** -4 * fl[0][1]), ("V", fl[1][0])]


def _mul(x, y):  # SU(2) matrices [[a, b], [-b*, a*]]
    return x[0] * y[0] - x[1] * y[1].conj(), x[0] * y[1] + x[1] * y[0].conj()


def _dag(x):
    return x[0].conj(), -x[1]


def _app(x, v):
    return x[0] * v[0] + x[1] * v[1], -x[1].conj() * v[0] + x[0].conj() * v[1]


def _sh(x, s, d):
    return tuple(s(y, d) for y in x)


class _SU2(_U1):
    def __init__(self, case, N, gS=G_SU2):
        self.dx, self.fm2, self.gS = _dx(case, N), (F_STAR_D / M_PL) ** 2, gS

    def parts(self, f):
        q = f[10:]
        U = [(torch.complex(q[4 * i], q[4 * i + 3]), torch.complex(q[4 * i + 2], q[4 * i + 1])) for i in range(3)]
        return f[0], torch.complex(f[1], f[2]), (torch.complex(f[3], f[4]), torch.complex(f[5], f[6])), f[7:10], U

    def forward(self, phi, D, A, U):
        u = self.links(A, G_U1_SU2)
        return ([u[d] * _up(phi, d) for d in range(3)],
                [tuple(u[d] * x for x in _app(U[d], _sh(D, _up, d))) for d in range(3)], u)

    def plaq(self, U, i, j):
        return _mul(_mul(_mul(U[i], _sh(U[j], _up, i)), _dag(_sh(U[i], _up, j))), _dag(U[j]))

    def kernel(self, f, a):
        S, phi, D, A, U = self.parts(f)
        dx, dx2 = self.dx, self.dx ** 2
        wC, wD, u = self.forward(phi, D, A, U)
        nD2, nC2 = _abs2(D[0]) + _abs2(D[1]), _abs2(phi)
        K = [a ** 2 * _lapl(S, dx) - a ** 4 * 2 * Q_GH * nD2 * S]
        lc = sum(wC[d] + _dn(u[d].conj() * phi, d) for d in range(3)) - 6 * phi
        kc = a ** 2 * lc / dx2 - a ** 4 / 2 * 4 * Q_GH * nD2 * phi
        back = [_sh(tuple(u[d].conj() * x for x in _app(_dag(U[d]), D)), _dn, d) for d in range(3)]
        m = 4 * nD2 + 2 * Q_GH * S ** 2 + 4 * Q_GH * nC2
        kd = [a ** 2 * (sum(wD[d][c] + back[d][c] for d in range(3)) - 6 * D[c]) / dx2 - a ** 4 / 2 * m * D[c] for c in range(2)]
        K += [kc.real, kc.imag, kd[0].real, kd[0].imag, kd[1].real, kd[1].imag]
        curl = self.curl(A)
        for i in range(3):
            J = (wC[i].conj() * phi).imag + (wD[i][0].conj() * D[0] + wD[i][1].conj() * D[1]).imag
            K.append(curl[i] - a ** 2 * 2 / dx * G_U1_SU2 * J)
        for i in range(3):
            g = [0, 0, 0]
            for j in range(3):
                if j != i:
                    P = self.plaq(U, i, j)
                    V = _sh(U[j], _up, i)  # U_i(x) U_j(x+i-j)^+ U_i(x-j)^+ U_j(x-j)
                    B = _mul(_mul(_mul(U[i], _dag(_sh(V, _dn, j))), _dag(_sh(U[i], _dn, j))), _sh(U[j], _dn, j))
                    g = [g[0] + P[1].imag + B[1].imag, g[1] + P[1].real + B[1].real, g[2] + P[0].imag + B[0].imag]
            sig = [(1j * D[1], 1j * D[0]), (D[1], -D[0]), (1j * D[0], -1j * D[1])]
            for c in range(3):
                J = 0.5 * self.gS * (wD[i][0].conj() * sig[c][0] + wD[i][1].conj() * sig[c][1]).real
                K.append(-g[c] / (dx ** 3 * self.gS) - a ** 2 / dx * J)
        return K

    def drift(self, f, p, aS, h):
        out = [x + h * aS ** -2 * y for x, y in zip(f[:7], p[:7])] + [x + h * y for x, y in zip(f[7:10], p[7:10])]
        for i in range(3):
            e = _qexp([h * self.dx * self.gS * y for y in p[10 + 3 * i:13 + 3 * i]])
            q = f[10 + 4 * i:14 + 4 * i]
            r = _mul((torch.complex(e[0], e[3]), torch.complex(e[2], e[1])),
                     (torch.complex(q[0], q[3]), torch.complex(q[2], q[1])))
            out += [r[0].real, r[1].imag, r[1].real, r[0].imag]
        return out

    def momenta(self, p):
        s = lambda i, j: sum(_mean(x ** 2) for x in p[i:j])  # noqa: E731
        return [s(0, 1), s(1, 3), s(3, 7), s(7, 10), 4 * s(10, 19)]

    def fields(self, f):
        S, phi, D, A, U = self.parts(f)
        wC, wD, _ = self.forward(phi, D, A, U)
        dx2 = self.dx ** 2
        gS = sum(_mean((_up(S, d) - S) ** 2) for d in range(3)) / dx2
        gC = sum(_mean(_abs2(wC[d] - phi)) for d in range(3)) / dx2
        gD = sum(_mean(_abs2(wD[d][c] - D[c])) for d in range(3) for c in range(2)) / dx2
        bG = sum(_mean(2 - 2 * self.plaq(U, i, j)[0].real) for i, j in ((1, 0), (2, 0), (2, 1)))
        nD2 = _abs2(D[0]) + _abs2(D[1])
        V = [_mean(nD2 ** 2), Q_GH * _mean(nD2 * S ** 2), 2 * Q_GH * _mean(nD2 * _abs2(phi))]
        return [gS, gC, gD, self.b2(A), 4 / (dx2 ** 2 * self.gS ** 2) * bG], V

    def energies(self, pi2, fl, a):
        g = fl[0]
        return [("K", 0.5 * pi2[0] * a ** -6), ("G", 0.5 * g[0] * a ** -2), ("K", pi2[1] * a ** -6), ("G", g[1] * a ** -2),
                ("K", pi2[2] * a ** -6), ("G", g[2] * a ** -2), ("E", 0.5 * a ** -4 * pi2[3]), ("E", 0.5 * a ** -4 * g[3]),
                ("E", 0.5 * a ** -4 * pi2[4]), ("E", 0.5 * a ** -4 * g[4])] + [("V", v) for v in fl[1]]


class _Evolution:
    """A lattice (or a stack of equal ones) with its scale factor, from a = 1 with the Friedmann ȧ."""

    def __init__(self, m, f, p, case):
        self.m, self.f, self.p, self.dt = m, f, p, _dt(case)
        self.ws = {"LF": (), "VV2": (1.0,), "VV4": (W4[0], W4[1], W4[0])}[case["evolver"]]
        self.a = self.aS = torch.ones_like(m.momenta(p)[0])
        self.pi2, self.fl = m.momenta(p), m.fields(f)
        self.pi2S = self.pi2
        rho = sum(v for _, v in m.energies(self.pi2, self.fl, self.a))
        self.aD = (self.a ** 4 / 3 * m.fm2 * rho).sqrt()
        self.aDS = self.aD - self.dt / 2 * self.acc()
        self.synced = True

    def acc(self):
        w = {"K": -1.0, "G": 1.0, "E": 0.0, "V": 2.0}
        return self.a ** 3 / 3 * self.m.fm2 * sum(w[k] * v for k, v in self.m.energies(self.pi2, self.fl, self.a))

    def kick(self, h):
        self.p = [x + h * k for x, k in zip(self.p, self.m.kernel(self.f, self.a))]

    def step(self):
        m, dt = self.m, self.dt
        if not self.ws:  # leapfrog
            self.kick(dt / 2 if self.synced else dt)
            self.synced = False
            old, self.pi2S = self.pi2S, m.momenta(self.p)
            self.pi2 = [(x + y) / 2 for x, y in zip(old, self.pi2S)]
            self.aDS = self.aDS + dt * self.acc()
            a0, self.a = self.a, self.a + dt * self.aDS
            self.aS = (a0 + self.a) / 2
            self.f = m.drift(self.f, self.p, self.aS, dt)
            self.fl = m.fields(self.f)
            return
        for w in self.ws:
            h = w * dt / 2
            aD = self.aD + h * self.acc()
            self.kick(h)
            a0, self.a = self.a, self.a + 2 * h * aD
            self.aS = (a0 + self.a) / 2
            self.f = m.drift(self.f, self.p, self.aS, 2 * h)
            self.fl = m.fields(self.f)
            self.kick(h)
            self.pi2 = m.momenta(self.p)
            self.aD = aD + h * self.acc()

    def sync(self):
        if not self.ws:
            self.kick(self.dt / 2)
            self.pi2 = self.m.momenta(self.p)
            self.aD = self.aDS + self.dt / 2 * self.acc()

    def energies(self):
        e = [v for _, v in self.m.energies(self.pi2, self.fl, self.a)]
        return torch.stack(e + [sum(e)])


class _Waves:
    """The five components u11, u12, u13, u22, u23 of the traceless u_ij, a leapfrog around the steps."""

    def __init__(self, ev):
        self.ev = ev
        self.u = [torch.zeros_like(ev.f[0]) for _ in range(5)]
        self.p = [torch.zeros_like(ev.f[0]) for _ in range(5)]

    def kick(self, w):
        ev, dx = self.ev, self.ev.m.dx
        g = [(_up(ev.f[0], d) - ev.f[0]) / dx for d in range(3)]
        third = (g[0] ** 2 + g[1] ** 2 + g[2] ** 2) / 3
        src = [g[0] ** 2 - third, g[0] * g[1], g[0] * g[2], g[1] ** 2 - third, g[1] * g[2]]
        self.p = [p + w * ev.dt * ev.a ** 2 * (_lapl(u, dx) + 2 * s) for p, u, s in zip(self.p, self.u, src)]

    def drift(self):
        self.u = [u + self.ev.aS ** -2 * self.ev.dt * p for u, p in zip(self.u, self.p)]


def _exact_gradient(case, f, p):
    from torch.utils.checkpoint import checkpoint

    f, p = f.requires_grad_(), p.requires_grad_()
    c = torch.tensor([1.0, G_U1], dtype=torch.float64, device="cuda", requires_grad=True)
    ev = _Evolution(_U1(case, case["N"], c[0], c[1]), list(f), list(p), case)
    names = ("f", "p", "a", "aD", "aS", "aDS", "pi2", "pi2S", "fl")

    def step(c, synced, *state):
        ev.m = _U1(case, case["N"], c[0], c[1])
        ev.synced = synced
        for k, v in zip(names, state):
            setattr(ev, k, v)
        ev.step()
        return tuple(getattr(ev, k) for k in names)

    state = tuple(getattr(ev, k) for k in names)
    flat, spec = torch.utils._pytree.tree_flatten(state)
    for i in range(case["steps"]):
        def one(c, *flat, synced=i == 0):
            return tuple(torch.utils._pytree.tree_flatten(step(c, synced, *torch.utils._pytree.tree_unflatten(list(flat), spec)))[0])

        flat = checkpoint(one, c, *flat, use_reentrant=False)
    for k, v in zip(names, torch.utils._pytree.tree_unflatten(list(flat), spec)):
        setattr(ev, k, v)
    ev.m = _U1(case, case["N"], c[0], c[1])
    ev.sync()
    e = ev.energies()
    obs = (e[2] + e[3]) / e[-1]
    gf, gp, gc = torch.autograd.grad(obs, (f, p, c))
    return {"observable": obs.detach()[None], "fields_bar": gf, "momenta_bar": gp, "couplings": gc}


def _exact_tangent(case, f, p):
    """The evolution on dual numbers along g_SU2, with the momenta's tangent that prepare() gives."""
    import torch.autograd.forward_ad as fwd

    with fwd.dual_level():
        one = torch.ones((), dtype=torch.float64, device="cuda")
        dp = torch.zeros_like(p)
        dp[10:] = -p[10:] / G_SU2
        m = _SU2(case, case["N"], fwd.make_dual(one * G_SU2, one))
        ev = _Evolution(m, list(f), [fwd.make_dual(x, y) for x, y in zip(p, dp)], case)
        for _ in range(case["steps"]):
            ev.step()
        ev.sync()
        e = ev.energies()
        obs = fwd.unpack_dual(sum(e[6:10]) / e[-1])
        val = lambda x: fwd.unpack_dual(x).primal  # noqa: E731
        dot = lambda x: torch.zeros_like(x) if fwd.unpack_dual(x).tangent is None else fwd.unpack_dual(x).tangent  # noqa: E731
        both = lambda g, v: torch.stack([g(x) for x in v])  # noqa: E731
        return {"fields": both(val, ev.f), "momenta": both(val, ev.p), "a": both(val, [ev.a, ev.aD]),
                "observable": torch.stack([obs.primal, obs.tangent]),
                "fields_dot": both(dot, ev.f), "momenta_dot": both(dot, ev.p)}


def exact(case, seed):
    kind, N = case["kind"], case["N"]
    with torch.set_grad_enabled(kind == "u1_gradient"):
        if kind == "u1_gradient":
            return _exact_gradient(case, *_start(case, N, seed))
        if kind == "ensemble":
            sizes = _member_sizes(case)
            f, p, a = [None] * len(sizes), [None] * len(sizes), [None] * len(sizes)
            for n in sorted(set(sizes)):
                at = [i for i, x in enumerate(sizes) if x == n]
                st = [_start(case, n, 1000 * seed + i) for i in at]
                ev = _Evolution(_Singlet(case, n), [torch.stack([x[0][0] for x in st])], [torch.stack([x[1][0] for x in st])], case)
                for _ in range(case["steps"]):
                    ev.step()
                for k, i in enumerate(at):
                    f[i], p[i], a[i] = ev.f[0][k].flatten(), ev.p[0][k].flatten(), torch.stack([ev.a[k], ev.aD[k]])
            return {"fields": torch.cat(f), "momenta": torch.cat(p), "a": torch.stack(a)}
        f, p = _start(case, N, seed)
        if kind == "su2_tangent":
            return _exact_tangent(case, f, p)
        m = {"u1": _U1, "su2": _SU2}.get(kind, _Singlet)(case, N)
        ev = _Evolution(m, list(f), list(p), case)
        gw = _Waves(ev) if kind == "gws" else None
        for i in range(case["steps"]):
            if gw:
                gw.kick(0.5 if i == 0 else 1.0)
            ev.step()
            if gw:
                gw.drift()
        ev.sync()
        if gw:
            gw.kick(0.5)
        out = {"fields": torch.stack(ev.f), "momenta": torch.stack(ev.p), "a": torch.stack([ev.a, ev.aD])}
        out["energies"] = ev.energies()
        if gw:
            out.update(spectra=None, gw=[torch.stack(gw.u), torch.stack(gw.p)])
        return out
