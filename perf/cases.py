"""Workloads of the time step, measured through the package's public entry points.

A case names one piece of work that a user's program has the library do: an output
interval of a simulation (K steps of a handle, then the fields and the diagnostics read
back), an ensemble's interval, a gradient call of a calibration loop, or a spectral solve
on the slab transform.  Grids, fields and step sizes are those of the decks in
``meumapps_ss_b200/configs.py`` and of the tests; a run of FP32-bulk fields is saved in
single precision, as its output files would be.

``listed`` gives the cases, ``draw`` more of the same ranges, ``prepare`` the handle and
inputs, ``run`` one pass, ``work`` what a pass cannot do without, ``exact`` the same
results in 64 bits with plain torch.
"""
import math

import numpy as np
import torch

from meumapps_ss_b200 import _lib
from meumapps_ss_b200 import configs as CF
from meumapps_ss_b200 import params as P

# 2^a 3^b lengths the generic path accepts, over the range its decks and tests use
LENGTHS = (24, 32, 36, 48, 54, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256)


def listed():
    return [
        # a driver coupled to another code: one step, then the fields are read (latency)
        dict(name="landau_32_f32_2v_1step", kind="landau", nx=32, ny=32, nz=32, nvar=2, f64=False, steps=1),
        # configuration 0: 64^3, one order parameter, plain FP64, one output interval
        dict(name="deck0_64_f64_1v", kind="landau", nx=64, ny=64, nz=64, nvar=1, f64=True, steps=100),
        # configuration 1, the headline: 128^3, three variants, FP32 bulk
        dict(name="deck1_128_f32_3v", kind="landau", nx=128, ny=128, nz=128, nvar=3, f64=False, steps=100),
        # configuration 3's mixture of sizes as an ensemble of 32
        dict(name="ensemble_32_f32", kind="ensemble", members=32, f64=False, steps=50),
        # configuration 2's heterogeneous fixed point on an HBM-sized grid
        dict(name="deck2_256_f32_4v", kind="hetero", nx=256, ny=256, nz=256, nvar=4, f64=False, steps=8),
        # the same model in FP64 on a box that is neither cubic nor a power of two
        dict(name="hetero_108x144x96_f64_2v", kind="hetero", nx=108, ny=144, nz=96, nvar=2, f64=True, steps=4),
        # the reference's own model at its usual size: three variants, heterogeneous cubic moduli
        dict(name="kks_128_f64_3v", kind="kks", nx=128, ny=128, nz=128, nvar=3, numel=1, f64=True, steps=5),
        # the reference's model on a small ragged box with two solutes (launches and waits count)
        dict(name="kks_48x36x54_f64_2sol", kind="kks", nx=48, ny=36, nz=54, nvar=1, numel=2, f64=True, steps=20),
        # twelve habit-plane variants, FP32 fields
        dict(name="kks_64_f32_12v", kind="kks", nx=64, ny=64, nz=64, nvar=12, numel=1, f64=False, steps=4),
        # nucleation stage: the reference's Langevin noise drawn before every step
        dict(name="kks_64_f64_noise", kind="noise", nx=64, ny=64, nz=64, nvar=1, numel=1, f64=True, steps=4),
        # configuration 4: loss and gradient of a calibration step (forward and backward)
        dict(name="adjoint_128_f32_1v", kind="adjoint", n=128, nvar=1, f64=False, steps=100, every=20),
        # screened Poisson solve on the slab-decomposed transform (forward and inverse), one rank
        dict(name="slab_512_f32", kind="slab", nx=512, ny=512, nz=512, f64=False),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi, cells):
    ok = [n for n in LENGTHS if lo <= n <= hi]
    while True:
        b = [rng.choice(ok) for _ in range(3)]
        if b[0] * b[1] * b[2] <= cells:
            return dict(nx=b[0], ny=b[1], nz=b[2])


def draw(rng):
    kind = rng.choice(("landau", "landau", "hetero", "hetero", "kks", "kks", "kks", "noise", "ensemble", "adjoint",
                       "slab"))
    f64 = rng.random() < 0.5
    if kind == "landau":
        n = rng.choice(CF.ENSEMBLE_SIZES)
        return dict(kind=kind, nx=n, ny=n, nz=n, nvar=rng.randint(1, 4), f64=f64, steps=_logint(rng, 1, 100))
    if kind == "hetero":
        return dict(kind=kind, **_box(rng, 32, 256, (64 if f64 else 128) * 256 * 256), nvar=rng.randint(1, 4), f64=f64,
                    steps=_logint(rng, 2, 6))
    if kind == "kks":
        numel = rng.choice((1, 1, 2))
        nvar = rng.choice((1, 3, 3, 12)) if numel == 1 else rng.choice((1, 3))
        return dict(kind=kind, **_box(rng, 24, 162, (48 ** 3 if nvar == 12 else 128 ** 3)), nvar=nvar, numel=numel,
                    f64=f64, steps=_logint(rng, 1, 10))
    if kind == "noise":
        return dict(kind=kind, **_box(rng, 24, 96, 64 ** 3), nvar=rng.choice((1, 3)), numel=1, f64=True,
                    steps=rng.randint(2, 4))
    if kind == "ensemble":
        return dict(kind=kind, members=_logint(rng, 6, 24), f64=f64, steps=_logint(rng, 5, 50))
    if kind == "adjoint":
        nvar = rng.randint(1, 2)
        return dict(kind=kind, n=rng.choice((32, 48, 64, 96) if nvar > 1 or f64 else (32, 64, 96, 128)), nvar=nvar,
                    f64=f64, steps=_logint(rng, 10, 60), every=rng.choice((5, 10, 20)))
    while True:
        b = [rng.choice((64, 72, 96, 108, 128, 144, 192, 216, 256, 288, 324, 384, 432, 512)) for _ in range(3)]
        if 128 ** 3 <= b[0] * b[1] * b[2] <= 256 * 512 * 512:
            return dict(kind="slab", nx=b[0], ny=b[1], nz=b[2], f64=f64)


# ------------------------------------------------------------------ decks and inputs
def _prec(case):
    return P.PREC_F64 if case["f64"] else P.PREC_F32


def _params(case):
    kind = case["kind"]
    if kind == "landau":
        # configurations 0 (one variant) and 1 on this grid
        nvar = case["nvar"]
        eig = [[0.01] * 3] if nvar == 1 else CF.tetragonal_variants(0.02, -0.005, nvar)
        return CF.landau_params(case["nx"], nvar, eig, dt=0.01 if nvar == 1 else 0.005, cross_w=0.0 if nvar == 1 else 0.5,
                                precision=_prec(case), ny=case["ny"], nz=case["nz"])
    if kind == "hetero":
        # configuration 2 on this grid
        return CF.landau_params(case["nx"], case["nvar"], CF.tetragonal_variants(0.015, -0.015 / 4, case["nvar"]),
                                dt=0.005, cross_w=0.5, coupling=P.EIG_H, elastic=P.ELAST_HETERO, ppt_scale=1.5,
                                el_tol=1e-8, precision=_prec(case), ny=case["ny"], nz=case["nz"])
    if kind == "adjoint":
        if case["nvar"] == 1:
            return CF.adjoint_config(case["n"], precision=_prec(case)).params
        return CF.landau_params(case["n"], case["nvar"], CF.tetragonal_variants(0.02, -0.005, case["nvar"]), dt=0.005,
                                cross_w=0.5, precision=_prec(case))
    noise_step = 10 ** 9 if kind == "noise" else 0
    deck = P.parse_input_txt(CF.kks_input_txt(case["nx"], case["nvar"], 1000, numel_in=case["numel"] + 1,
                                              noise_step=noise_step, ny=case["ny"], nz=case["nz"]))
    return P.kks_params(deck, precision=_prec(case), sym_var=CF.tetrahedral_rotations())


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _uniform(shape, g, lo, hi):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _nuclei(nvar, nz, ny, nx, g):
    """Smooth-edged precipitates of every variant: about one sphere per 24^3 cells, radii of
    3 to 7 cells, on a small background, each variant's order parameter in [0, 1]."""
    count = max(2, min(64, nx * ny * nz // 24 ** 3))
    u = torch.rand((count, 5), generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
    phi = _uniform((nvar, nz, ny, nx), g, 0.0, 0.01)
    ax = [torch.arange(n, device="cuda", dtype=torch.float64) for n in (nz, ny, nx)]
    for k in range(count):
        r = 3.0 + 4.0 * u[k, 3]
        d2 = 0
        for d, n in enumerate((nz, ny, nx)):
            q = (ax[d] - u[k, d] * n).abs()
            q = torch.minimum(q, n - q) ** 2
            d2 = d2 + q.reshape([-1 if e == d else 1 for e in range(3)])
        f = 0.5 * (1.0 - torch.tanh(d2.sqrt() - r))
        v = min(int(u[k, 4] * nvar), nvar - 1)
        phi[v] = torch.maximum(phi[v], f)
    return phi.clamp_(0.0, 1.0)


def _fields(case, seed):
    """(c, phi) as (ncomp, nz, ny, nx) FP64 tensors on the GPU."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "adjoint":
        n = (case["n"],) * 3
        return _uniform((1,) + n, g, 0.75, 0.85), _uniform((case["nvar"],) + n, g, -0.5, 0.5)
    n = (case["nz"], case["ny"], case["nx"])
    if kind == "landau":
        c0 = 0.15 if case["nvar"] == 1 else 0.2
        return _uniform((1,) + n, g, c0 - 0.01, c0 + 0.01), _uniform((case["nvar"],) + n, g, -0.001, 0.001)
    if kind == "hetero":
        return _uniform((1,) + n, g, 0.19, 0.21), _uniform((case["nvar"],) + n, g, -0.005, 0.005)
    phi = _nuclei(case["nvar"], *n, g)
    p = phi ** 3 * (6 * phi ** 2 - 15 * phi + 10)
    far, near = ((0.15, 0.55), (0.07, 0.20)), p.sum(0).clamp(max=1.0)
    c = torch.stack([a + (b - a) * near for a, b in far[:case["numel"]]])
    return c + _uniform(c.shape, g, -0.002, 0.002), phi


def _members(case):
    return CF.ensemble_config(case["members"], precision=_prec(case))


def _pinned(n):
    t = torch.empty(n, dtype=torch.float64, pin_memory=True)
    return t, t.numpy()


def _host(soa):
    """Fortran-layout host copy (component fastest) in page-locked memory."""
    f = soa.movedim(0, -1).contiguous().reshape(-1)
    t, a = _pinned(f.numel())
    t.copy_(f)
    return t, a


class _Out:
    """Page-locked output arrays of a run and, for FP32-bulk runs, their single-precision form."""

    def __init__(self, sizes, f64):
        self.t, self.a = {}, {}
        for k, n in sizes.items():
            self.t[k], self.a[k] = _pinned(n)
        self.single = None if f64 else {k: torch.empty(n, dtype=torch.float32) for k, n in sizes.items()}

    def saved(self):
        if self.single is None:
            return dict(self.t)
        for k, s in self.single.items():
            s.copy_(self.t[k])
        return dict(self.single)


def _rows(n):
    rows = (P.MeuDiag * n)()
    return rows, np.frombuffer(rows, dtype=np.dtype(P.MeuDiag))


ENERGY = ("fint", "fw", "fch", "elen", "etot")
STATS = ("cmin", "cmax", "phimax", "solid_now")


def _diag(view, f64):
    t = np.float64 if f64 else np.float32
    return {"energy": np.stack([view[k] for k in ENERGY], 1).astype(t),
            "stats": np.concatenate([np.stack([view[k] for k in STATS], 1), view["cavg"][:, :1]], 1).astype(t)}


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    from meumapps_ss_b200.sim import Ensemble, Simulation

    kind, f64 = case["kind"], case["f64"]
    if kind == "slab":
        from meumapps_ss_b200.slab_fft import SlabFFT
        rt = torch.float64 if f64 else torch.float32
        fft = SlabFFT(case["nx"], case["ny"], case["nz"], precision=_prec(case))
        real = torch.randn(fft.real_shape, generator=_gen(seed), device="cuda", dtype=rt)
        return dict(case=case, fft=fft, real=real, solve=_screened(case).to(rt))
    if kind == "ensemble":
        w = _members(case)
        e = Ensemble([m.params for m in w])
        cells = [m.params.nx ** 3 for m in w]
        g = _gen(seed)
        at = np.concatenate([[0], np.cumsum(cells)])
        c = torch.cat([_uniform((n,), g, m.c0 - m.c_amp, m.c0 + m.c_amp) for m, n in zip(w, cells)])
        f = _uniform((int(at[-1]),), g, -0.001, 0.001)
        (_, hc), (_, hf) = _host(c[None]), _host(f[None])
        for m in range(len(w)):
            e.set_fields_fortran(m, hc[at[m]:at[m + 1]], hf[at[m]:at[m + 1]])
        rows, view = _rows(len(w) * case["steps"])
        return dict(case=case, ens=e, at=[int(x) for x in at], rows=rows, view=view,
                    out=_Out({"c": int(at[-1]), "phi": int(at[-1])}, f64))
    p = _params(case)
    c, f = _fields(case, seed)
    (kc, hc), (kf, hf) = _host(c), _host(f)
    sim = Simulation(p)
    n3 = p.nx * p.ny * p.nz
    s = dict(case=case, sim=sim)
    if kind == "adjoint":
        g = _gen(seed + 1)
        tc, tf = c + _uniform(c.shape, g, -0.01, 0.01), 0.9 * f
        pin = [torch.empty(t.shape, dtype=torch.float64, pin_memory=True).copy_(t) for t in (tc, tf)]
        s.update(keep=(kc, kf, pin), hc=hc, hf=hf, tc=pin[0].numpy(), tf=pin[1].numpy(),
                 single=torch.empty(f.shape, dtype=torch.float32))
        return s
    sim.set_fields_fortran(hc, hf)
    sizes = {"c": c.numel(), "phi": f.numel()}
    if kind != "landau":
        sizes["el"] = n3
    rows, view = _rows(case["steps"])
    s.update(rows=rows, view=view, out=_Out(sizes, f64))
    if kind == "noise":
        s["rng"] = _lib.Ran2(-(1 + seed % 100000))
    return s


def run(state):
    case = state["case"]
    kind, f64 = case["kind"], case["f64"]
    if kind == "slab":
        k = state["fft"].forward(state["real"])
        k.mul_(state["solve"])
        return {"solution": state["fft"].inverse(k)}
    if kind == "ensemble":
        e, at, out = state["ens"], state["at"], state["out"]
        e.run_into(case["steps"], state["rows"])
        for m in range(len(at) - 1):
            e.get_fields_fortran(m, out.a["c"][at[m]:at[m + 1]], out.a["phi"][at[m]:at[m + 1]])
        return {**out.saved(), **_diag(state["view"], f64)}
    sim = state["sim"]
    if kind == "adjoint":
        sim.set_fields_fortran(state["hc"], state["hf"])
        loss, grads, field = sim.adjoint(case["steps"], case["every"], state["tc"], state["tf"])
        field = torch.from_numpy(np.ascontiguousarray(field)).reshape(state["single"].shape)
        t = np.float64 if f64 else np.float32
        return {"loss": np.array([loss], dtype=t), "grads": [np.array([grads[k]], dtype=t) for k in sorted(grads)],
                "dphi0": field if f64 else state["single"].copy_(field)}
    if kind == "noise":
        # the draws' host generator advances with the simulation
        _run_noise(sim, case["steps"], state)
    else:
        sim.run_into(case["steps"], state["rows"])
    out = state["out"]
    sim.get_fields_fortran(out.a["c"], out.a["phi"], out.a.get("el"))
    got = {**out.saved(), **_diag(state["view"], f64)}
    if f64 and kind != "landau":
        got["el_iters"] = state["view"]["el_iters"].copy()
    return got


def _run_noise(sim, steps, state):
    got = sim.run_noise(steps, state["rng"].s, 1.0e-3)
    for k in ("el_iters",) + ENERGY + STATS + ("cavg",):
        state["view"][k] = got[k]


# ------------------------------------------------------------------ work
def _fft_flops(nx, ny, nz):
    n = nx * ny * nz
    return 2.5 * n * math.log2(n)


def work(case):
    """Compulsory bytes: the fields (and the spectral or elastic state) of every step read and
    written once in the field precision, plus the output copies; the flops of the transforms
    that the step's formulas ask for."""
    r = 8 if case["f64"] else 4
    kind = case["kind"]
    if kind == "slab":
        n = case["nx"] * case["ny"] * case["nz"]
        nk = (case["nx"] // 2 + 1) * case["ny"] * case["nz"]
        # real in, spectrum out; spectrum in and out of the solve with its factors; spectrum in, real out
        return {"bytes": r * (2.0 * n + 9.0 * nk), "flops": 2 * _fft_flops(case["nx"], case["ny"], case["nz"]) + 2.0 * nk}
    if kind == "ensemble":
        cells = [m.params.nx ** 3 for m in _members(case)]
        n, k = sum(cells), case["steps"]
        return {"bytes": k * 2.0 * 2 * r * n + 8.0 * 2 * n,
                "flops": k * sum(7.0 * 2.5 * m * math.log2(m) for m in cells)}
    if kind == "adjoint":
        n, v, k = case["n"] ** 3, case["nvar"], case["steps"]
        # forward, recomputation and reverse: the state in and out of each step, the recorded state in
        return {"bytes": k * 3.0 * 2 * (v + 1) * r * n + 8.0 * (2 * (v + 1) + v) * n,
                "flops": k * 3.0 * (4 * v + 2) * _fft_flops(case["n"], case["n"], case["n"])}
    nx, ny, nz, v, k = case["nx"], case["ny"], case["nz"], case["nvar"], case["steps"]
    n, ft = nx * ny * nz, _fft_flops(nx, ny, nz)
    if kind == "landau":
        return {"bytes": k * 2.0 * (v + 1) * r * n + 8.0 * (v + 1) * n, "flops": k * (5.0 * v + 2) * ft}
    e = case.get("numel", 1)
    # heterogeneous elasticity: 4 fixed-point iterations at least, each 6 transforms each way,
    # the strain in and out of each iteration once
    local = (3 * v + 2) * ft if kind == "hetero" else (7 * v + 5 * e) * ft
    return {"bytes": k * (2.0 * (v + e) + 4 * 2.0 * 6) * r * n + 8.0 * (v + e + 1) * n, "flops": k * (local + 48 * ft)}


# ------------------------------------------------------------------ 64-bit results
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Grid:
    """f_trans / inv_trans and k-vectors: a = 2 pi m / N with m in (-N/2, N/2], b = a with the
    Nyquist index zeroed; spectra [kz][ky][kx], kx in [0, N/2]."""

    def __init__(self, nx, ny, nz):
        self.s, self.n3 = (nz, ny, nx), nx * ny * nz
        self.a, self.b = [], []
        for d, (n, half) in enumerate(((nx, True), (ny, False), (nz, False))):
            m = torch.arange(n // 2 + 1 if half else n, dtype=torch.float64, device=_device())
            a = 2 * math.pi / n * torch.where(m <= n // 2, m, m - n)
            b = torch.where(2 * m == n, torch.zeros_like(a), a)
            shape = [1, 1, 1]
            shape[2 - d] = -1
            self.a.append(a.reshape(shape))
            self.b.append(b.reshape(shape))
        self.k2 = self.a[0] ** 2 + self.a[1] ** 2 + self.a[2] ** 2

    def f(self, x):
        return torch.fft.rfftn(x) / self.n3

    def i(self, x):
        return torch.fft.irfftn(x, s=self.s) * self.n3

    def kappa(self, g, sq):
        """k.kappa.k with `sq` on the diagonal and b off it (g: 9 values, column-major)."""
        b = self.b
        return (g[0] * sq[0] ** 2 + g[4] * sq[1] ** 2 + g[8] * sq[2] ** 2 + (g[3] + g[1]) * b[0] * b[1]
                + (g[7] + g[5]) * b[1] * b[2] + (g[2] + g[6]) * b[2] * b[0])

    def inverse_q(self, c6):
        """The 6 entries (xx, yy, zz, yz, xz, xy) of Q(k)^-1 of a cubic stiffness (C11, C12, C44)."""
        c11, c12, c44 = c6
        a, b = self.a, self.b
        own, off = -c11, -c44
        q = [own * a[d] ** 2 + off * (self.k2 - a[d] ** 2) for d in range(3)]
        yz, xz, xy = (-(c12 + c44) * b[i] * b[j] for i, j in ((1, 2), (0, 2), (0, 1)))
        m = [q[1] * q[2] - yz * yz, q[0] * q[2] - xz * xz, q[0] * q[1] - xy * xy, xy * xz - q[0] * yz,
             xy * yz - q[1] * xz, xz * yz - q[2] * xy]
        det = q[0] * m[0] + xy * m[5] + xz * m[4]
        det[0, 0, 0] = 1.0
        out = [e / det for e in m]
        for e in out:
            e[0, 0, 0] = 0.0
        return out


def _mul_sym(q, r):
    return [q[0] * r[0] + q[5] * r[1] + q[4] * r[2], q[5] * r[0] + q[1] * r[1] + q[3] * r[2],
            q[4] * r[0] + q[3] * r[1] + q[2] * r[2]]


def _cubic(p, name, n):
    m = p.matrix(name, n, 6)
    return m[0, 0], m[0, 1], m[3, 3]


def _apply(c, e):
    """A cubic stiffness or compliance (its 3 constants, numbers or fields) times a Voigt vector."""
    t = c[1] * (e[0] + e[1] + e[2])
    return [(c[0] - c[1]) * e[i] + t for i in range(3)] + [c[2] * e[i] for i in range(3, 6)]


def _cubic_inverse(c):
    s, d = c[0] + 2 * c[1], c[0] - c[1]
    return (c[0] + c[1]) / (s * d), -c[1] / (s * d), 1.0 / c[2]


def _kf(g, s):
    """i (b . S) of the three rows of a symmetric Voigt tensor field of spectra."""
    b = g.b
    return [1j * (b[0] * s[0] + b[1] * s[5] + b[2] * s[4]), 1j * (b[0] * s[5] + b[1] * s[1] + b[2] * s[3]),
            1j * (b[0] * s[4] + b[1] * s[3] + b[2] * s[2])]


def _strain(g, u):
    b = g.b
    return [1j * b[0] * u[0], 1j * b[1] * u[1], 1j * b[2] * u[2], 1j * (b[1] * u[2] + b[2] * u[1]),
            1j * (b[0] * u[2] + b[2] * u[0]), 1j * (b[0] * u[1] + b[1] * u[0])]


class _Elastic:
    """The elastic fixed point and its energies on cubic moduli (ModElastic.f:105-691)."""

    def __init__(self, p, g, phase):
        self.p, self.g, self.phase = p, g, phase
        self.cel = [_cubic(p, "cela", n) for n in range(p.numph)]
        self.sel = [_cubic(p, "sela", n) for n in range(p.numph)]
        self.tr = [[p.trans_ppt[v][m] for m in range(6)] for v in range(p.nvar)]
        self.eng = [[t[m] * (1 if m < 3 else 2) for m in range(6)] for t in self.tr]
        self.q = g.inverse_q(self.cel[1])
        self.u, self.gam = None, None

    def mix(self, pphi, w):
        return [sum(pphi[v] * self.sel[n][k] for v, n in enumerate(self.phase)) + w * self.sel[0][k] for k in range(3)]

    def solve(self, r):
        return _mul_sym(self.q, r)

    def step(self, pphi, phi, first):
        p, g = self.p, self.g
        if first:
            ph = [g.f(x) for x in pphi]
            sig0 = [_apply(self.cel[n], self.eng[v]) for v, n in enumerate(self.phase)]
            self.u = self.solve(_kf(g, [sum(ph[v] * sig0[v][m] for v in range(p.nvar)) for m in range(6)]))
            self.gam = [g.i(x) for x in _strain(g, self.u)]
        psum = sum(pphi)
        cm = _cubic_inverse(self.mix(pphi, torch.where(psum < 1, 1 - psum, torch.zeros_like(psum))))
        e0 = [sum(pphi[v] * self.eng[v][m] for v in range(p.nvar)) for m in range(6)]
        newfac, cfac, niter, total, old = 0.5, 1.0, 0, 0, None
        done = False
        while True:
            niter, total = niter + 1, total + 1
            ca, cb = _apply(self.cel[1], self.gam), _apply(cm, [e0[m] - cfac * self.gam[m] for m in range(6)])
            u = self.solve(_kf(g, [g.f(cfac * ca[m] + cb[m]) for m in range(6)]))
            ui, uo = [g.i(x) for x in u], [g.i(x) for x in self.u]
            ratio = [float(((x - y) ** 2).sum() / (y ** 2).sum()) for x, y in zip(ui, uo)]
            self.u, self.gam = u, [g.i(x) for x in _strain(g, u)]
            done = done or all(r < p.el_tol for r in ratio)
            if niter > 1 and not done and any(r > o for r, o in zip(ratio, old)):
                cfac, newfac, niter, done = cfac * newfac, newfac * 0.5, 0, False
                continue
            old = ratio
            done = done or niter == p.el_max_iter
            if not done or niter < p.el_min_iter:
                continue
            if cfac < 1 - 1e-6:
                cfac, niter, done = min(cfac + 0.1, 1.0), 0, False
                continue
            break
        ce = _cubic_inverse(self.mix(pphi, 1 - psum))
        sig = _apply(ce, [self.gam[m] - e0[m] for m in range(6)])
        dens = lambda s: 0.5 * sum(x * y for x, y in zip(sig, _apply(s, sig)))  # noqa: E731
        mat = dens(self.sel[0])
        en, grad = (1 - psum) * mat, []
        for v, n in enumerate(self.phase):
            t, f = self.tr[v], phi[v]
            if self.p.model == P.MODEL_KKS and not sum(t) > float(np.float32(1e-9)):
                grad.append(torch.zeros_like(f))
                continue
            ppt = dens(self.sel[n])
            en = en + ppt * pphi[v]
            s = sum(sig[m] * t[m] * (1 if m < 3 else 2) for m in range(6))
            grad.append(30 * f ** 2 * (f ** 2 - 2 * f + 1) * (mat - ppt - s))
        return en, grad, total


def _col(x):
    return torch.stack(x, -1).reshape(-1)


def _stats(c, phi, kks):
    solid = phi.clamp(min=0).sum() if kks else (phi ** 2).sum()
    n3 = c[0].numel()
    return [min(1.0, float(c.min())), max(0.0, float(c.max())), max(0.0, float(phi.max())), float(solid) / n3,
            float(c[0].sum()) / n3]


class _Landau:
    """The Landau step (functional of include/meu.h); scales for the calibration parameters."""

    def __init__(self, p, energy=True):
        self.p, self.energy = p, energy
        self.g = g = _Grid(p.nx, p.ny, p.nz)
        self.het = p.elastic == P.ELAST_HETERO
        self.den = [g.kappa([p.grad_coeff[v][i] for i in range(9)], g.a) for v in range(p.nvar)]
        if self.het:
            self.el = _Elastic(p, g, [1] * p.nvar)
            return
        cel = _cubic(p, "cela", 1)
        self.eng = [[p.trans_ppt[v][m] * (1 if m < 3 else 2) for m in range(6)] for v in range(p.nvar)]
        self.sig0 = [_apply(cel, e) for e in self.eng]
        self.cel, self.q = cel, g.inverse_q(cel)
        b = g.b
        self.sb = [[s[0] * b[0] + s[5] * b[1] + s[4] * b[2], s[5] * b[0] + s[1] * b[1] + s[3] * b[2],
                    s[4] * b[0] + s[3] * b[1] + s[2] * b[2]] for s in self.sig0]
        self.A = [[sum(x * y for x, y in zip(self.eng[v], self.sig0[w])) for w in range(p.nvar)] for v in range(p.nvar)]

    def step(self, c, eta, first=True, beta=1.0, kc=None, L=None, M=None, alpha=1.0):
        p, g, V = self.p, self.g, self.p.nvar
        kc, L, M = (p.kappa_c if kc is None else kc), (p.b_mob if L is None else L), (p.cmobs[0] if M is None else M)
        e2 = [x * x for x in eta]
        s2 = sum(e2)
        mu = g.f(p.lan_a * (c - p.lan_c1) - 0.5 * p.lan_b * s2)
        ck, ek = g.f(c), [g.f(x) for x in eta]
        info = None
        if self.het:
            th = [x ** 3 * (6 * x * x - 15 * x + 10) for x in eta]
            en, grad, iters = self.el.step(th, eta, first)
        else:
            tk = [g.f(x) for x in e2]
            r = [1j * sum(tk[v] * self.sb[v][d] for v in range(V)) for d in range(3)]
            u = _mul_sym(self.q, r)
            pot = [g.i(1j * sum(self.sb[v][d] * u[d] for d in range(3))) for v in range(V)]
            grad = [-2 * eta[v] * alpha ** 2 * (pot[v] - sum(self.A[v][w] * e2[w] for w in range(V))) for v in range(V)]
        if self.energy:
            s4, s6 = sum(x * x for x in e2), sum(x ** 3 for x in e2)
            fch = (0.5 * p.lan_a * (c - p.lan_c1) ** 2 + 0.5 * p.lan_b * (p.lan_c2 - c) * s2 - 0.25 * p.lan_c * s4
                   + p.lan_d / 6 * s6 + p.cross_w * (s2 * s2 - s4)).sum()
            w = torch.full((p.nx // 2 + 1,), 2.0, dtype=torch.float64, device=c.device)
            w[0] = w[-1] = 1.0
            ab = lambda x: x.real ** 2 + x.imag ** 2  # noqa: E731
            fint = (0.5 * w * kc * (g.b[0] ** 2 + g.b[1] ** 2 + g.b[2] ** 2) * ab(ck)).sum()
            for v in range(V):
                fint = fint + (0.5 * w * g.kappa([p.grad_coeff[v][i] for i in range(9)], g.b) * ab(ek[v])).sum()
            if self.het:
                elen = en.sum()
            else:
                e = [g.i(x) for x in _strain(g, u)]
                e = [e[m] - sum(e2[v] * self.eng[v][m] for v in range(V)) for m in range(6)]
                elen = 0.5 * sum((x * y).sum() for x, y in zip(e, _apply(self.cel, e)))
            row = [float(fint) * g.n3, 0.0, float(fch), float(elen)]
            info = dict(energy=row + [sum(row)], el=en if self.het else None, iters=iters if self.het else 0)
        dm, dl = p.dt * M, p.dt * L
        ck = (ck - dm * g.k2 * mu) / (1 + dm * kc * g.k2 ** 2)
        new = []
        for v in range(V):
            gv = (p.lan_b * (p.lan_c2 - c) * eta[v] - p.lan_c * eta[v] ** 3 + p.lan_d * eta[v] ** 5
                  + 4 * p.cross_w * eta[v] * (s2 - e2[v]) + grad[v])
            new.append(g.i((ek[v] - dl * g.f(gv)) / (1 + dl * beta * self.den[v])))
        return g.i(ck), new, info


class _Kks:
    """The reference's KKS step without noise (Multi_MEUMAPPS.f:575-1043)."""

    def __init__(self, p):
        self.p = p
        self.g = _Grid(p.nx, p.ny, p.nz)
        self.phase = [n for n in range(1, p.numph) for _ in range(p.nvar_ph[n])]
        self.el = _Elastic(p, self.g, self.phase)

    def step(self, cons, phi, first):
        p, g, V, E, H = self.p, self.g, self.p.nvar, self.p.numel, self.p.numph
        G = lambda j, n: p.gparams[n][j]  # noqa: E731  (0-based row, 0-based phase)
        gc = [[p.grad_coeff[v][i] for i in range(9)] for v in range(V)]
        fk = [g.f(x) for x in phi]
        grad = [[g.i(1j * g.b[d] * x) for d in range(3)] for x in fk]
        kap = [g.kappa(gc[v], g.a) for v in range(V)]
        lap = [g.i(-kap[v] * fk[v]) for v in range(V)]
        pl = [f ** 3 * (6 * f ** 2 - 15 * f + 10) for f in phi]
        ppr = [30 * f ** 2 * (f ** 2 - 2 * f + 1) for f in phi]
        pph = [1 - sum(pl)] + [sum(pl[v] for v in range(V) if self.phase[v] == n) for n in range(1, H)]
        sq = sum(f ** 2 for f in phi)
        well = [sum(f ** 2 * (sq - f ** 2) for f in phi)]
        well += [sum(phi[v] ** 2 * (1 - phi[v]) ** 2 for v in range(V) if self.phase[v] == n) for n in range(1, H)]
        # interface compositions: equal potentials, mixture rule
        z = E * H
        Z = torch.zeros((g.n3, z, z), dtype=torch.float64, device=phi.device)
        R = torch.zeros((g.n3, z), dtype=torch.float64, device=phi.device)
        for e in range(E):
            for n in range(H - 1):
                i = (H - 1) * e + n
                Z[:, i, H * e + n], Z[:, i, H * e + n + 1] = G(e, n), -G(e, n + 1)
                R[:, i] = G(e, n) * G(E + 1 + e, n) - G(e, n + 1) * G(E + 1 + e, n + 1)
            i = z - E + e
            R[:, i] = cons[e].reshape(-1)
            for n in range(H):
                Z[:, i, H * e + n] = pph[n].reshape(-1)
        X = torch.linalg.solve(Z, R[..., None])[..., 0]
        x = [[X[:, H * e + n].reshape(g.s) for n in range(H)] for e in range(E)]
        gib = [sum(G(e, n) * (x[e][n] - G(E + 1 + e, n)) ** 2 for e in range(E)) + G(E, n) for n in range(H)]
        mu = [2 * G(e, 0) * (x[e][0] - G(E + 1 + e, 0)) for e in range(E)]
        fch = sum(pph[n] * gib[n] for n in range(H)).sum()
        fw = sum(p.wellph[n] * well[n] for n in range(H)).sum()
        fint, flux, fg = 0.0, [[0.0] * 3 for _ in range(E)], []
        for v in range(V):
            n, f, (gx, gy, gz), c = self.phase[v], phi[v], grad[v], gc[v]
            fint = fint + 0.5 * (c[0] * gx * gx + c[4] * gy * gy + c[8] * gz * gz + (c[3] + c[1]) * gx * gy
                                 + (c[6] + c[2]) * gx * gz + (c[7] + c[5]) * gy * gz).sum()
            t = gib[n] - gib[0]
            for e in range(E):
                xd = x[e][0] - x[e][n]
                t = t + mu[e] * xd
                for d in range(3):
                    flux[e][d] = flux[e][d] + ppr[v] * xd * grad[v][d]
            fg.append(t * ppr[v] + 2 * p.wellph[n] * f * (1 - f) * (1 - 2 * f) + 4 * p.wellph[0] * f * (sq - f ** 2))
        fd = []
        for j in range(V):
            acc, cnt = torch.zeros_like(phi[j]), torch.ones_like(phi[j])
            for i in range(V):
                if i != j:
                    on = (phi[j] > 0) & (phi[i] > 0)
                    acc, cnt = acc + torch.where(on, fg[i] - lap[i], torch.zeros_like(acc)), cnt + on
            fd.append(fg[j] - acc / cnt)
        en, eg, iters = self.el.step(pl, phi, first)
        new_c = []
        for e in range(E):
            dm = p.dt * p.cmobs[e]
            div = 1j * sum(g.b[d] * g.f(flux[e][d]) for d in range(3))
            new_c.append(g.i((g.f(cons[e]) + dm * div) / (1 + dm * g.k2)))
        dl = p.dt * p.b_mob
        new = [g.i((fk[v] - dl * g.f(fd[v] + eg[v])) / (1 + dl * kap[v])).clamp(0.0, 1.0) for v in range(V)]
        row = [float(fint), float(fw), float(fch), float(en.sum())]
        return torch.stack(new_c), torch.stack(new), dict(energy=row + [sum(row)], el=en, iters=iters)


def _march(stepper, c, phi, steps, kks):
    energy, stats, iters, info = [], [], [], None
    for s in range(steps):
        if kks:
            c, phi, info = stepper.step(c, phi, s == 0)
        else:
            cn, new, info = stepper.step(c[0], [x for x in phi], s == 0)
            c, phi = cn[None], torch.stack(new)
        energy.append(info["energy"])
        stats.append(_stats(c, phi, kks))
        iters.append(info["iters"])
    return c, phi, np.array(energy), np.array(stats), np.array(iters), info["el"]


def _screened(case):
    g = _Grid(case["nx"], case["ny"], case["nz"])
    return 1.0 / (1.0 + g.k2)


def exact(case, seed):
    kind = case["kind"]
    if kind == "noise":
        return None  # the serial ran_2 stream takes minutes in plain Python
    if kind == "slab":
        g = _Grid(case["nx"], case["ny"], case["nz"])
        rt = torch.float64 if case["f64"] else torch.float32
        real = torch.randn(g.s, generator=_gen(seed), device="cuda", dtype=rt)
        return {"solution": g.i(g.f(real.double()) * _screened(case).to(rt).double())}
    if kind == "ensemble":
        w = _members(case)
        g = _gen(seed)
        cells = [m.params.nx ** 3 for m in w]
        c = [_uniform((n,), g, m.c0 - m.c_amp, m.c0 + m.c_amp) for m, n in zip(w, cells)]
        f = torch.split(_uniform((sum(cells),), g, -0.001, 0.001), cells)
        outs = []
        for m, ci, fi in zip(w, c, f):
            n = (1,) + (m.params.nx,) * 3
            outs.append(_march(_Landau(m.params), ci.reshape(n), fi.reshape(n), case["steps"], False))
        return {"c": torch.cat([o[0].reshape(-1) for o in outs]), "phi": torch.cat([o[1].reshape(-1) for o in outs]),
                "energy": np.concatenate([o[2] for o in outs]), "stats": np.concatenate([o[3] for o in outs])}
    p = _params(case)
    c, f = _fields(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed, p, c, f)
    kks = kind == "kks"
    c, f, energy, stats, iters, el = _march(_Kks(p) if kks else _Landau(p), c, f, case["steps"], kks)
    got = {"c": _col(list(c)), "phi": _col(list(f)), "energy": energy, "stats": stats}
    if kind != "landau":
        got["el"] = el.reshape(-1)
        if case["f64"]:
            got["el_iters"] = iters.astype(np.int32)
    return got


def _exact_adjoint(case, seed, p, c, f):
    """The gradient by torch's reverse mode, segment by segment (recomputed from checkpoints)."""
    from torch.utils.checkpoint import checkpoint

    gen = _gen(seed + 1)
    tc, tf = c + _uniform(c.shape, gen, -0.01, 0.01), 0.9 * f
    par = [torch.tensor(x, dtype=torch.float64, device=c.device, requires_grad=True)
           for x in (1.0, p.kappa_c, p.b_mob, p.cmobs[0], 1.0)]
    f0 = f.clone().requires_grad_(True)
    lan = _Landau(p, energy=False)

    def segment(c, f, n, *q):
        for _ in range(n):
            c, f, _ = lan.step(c, f, True, q[0], q[1], q[2], q[3], q[4])
            f = torch.stack(f)
        return c, f

    x, y, left = c[0], f0, case["steps"]
    while left:
        n = min(10, left)
        x, y = checkpoint(segment, x, y, n, *par, use_reentrant=False)
        left -= n
    loss = 0.5 / lan.g.n3 * (((y - tf) ** 2).sum() + ((x - tc[0]) ** 2).sum())
    loss.backward()
    names = ("beta_eta", "kappa_c", "L", "M", "alpha")
    grads = {k: q.grad.reshape(1) for k, q in zip(names, par)}
    return {"loss": loss.detach().reshape(1), "grads": [grads[k] for k in sorted(grads)], "dphi0": f0.grad}
