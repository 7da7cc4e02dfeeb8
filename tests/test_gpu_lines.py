"""The heterogeneous Landau and KKS steps on boxes whose sides reach every radix plan of the
compile-time line kernels (two and three stages, radices 4 to 16, the FP32 / FP64 tile widths)
and partial last tiles, against the oracle; and FP32 fields against FP64 on the same boxes."""
import numpy as np
import pytest

from helpers import kks_case
from meumapps_ss_b200 import configs as CF
from meumapps_ss_b200 import params as P

pytestmark = pytest.mark.gpu

# (nx, ny, nz): every length with a compile-time plan once as nz, most as ny, as nx and nx / 2
BOXES = [(8, 6, 16), (24, 16, 24), (36, 24, 32), (12, 32, 36), (48, 4, 48), (54, 36, 54), (16, 48, 64), (32, 9, 72),
         (64, 54, 8), (6, 64, 96), (72, 8, 108), (10 + 2, 72, 128), (96, 6, 144), (108, 96, 4), (8, 6, 162),
         (128, 8, 192), (144, 9, 216), (162, 108, 6), (6, 8, 256), (192, 12, 288), (8, 4, 324), (216, 8, 384),
         (256, 4, 432), (4, 6, 512), (288, 128, 3), (324, 144, 2), (384, 2, 162), (432, 192, 2), (512, 6, 4), (6, 216, 4)]


def _fields(p, seed):
    rng = np.random.default_rng(seed)
    s = (p.nz, p.ny, p.nx)
    return 0.8 + 0.05 * rng.uniform(-1, 1, (1,) + s), 0.5 * rng.uniform(-1, 1, (p.nvar,) + s)


def _run(p, c, e, steps):
    from meumapps_ss_b200.sim import Simulation
    with Simulation(p) as g:
        g.set_fields(c, e)
        d = g.run(steps)
        return d, g.get_fields()


@pytest.mark.parametrize("box", BOXES)
def test_hetero_box_matches_oracle(oracle, box):
    nx, ny, nz = box
    p = CF.landau_params(nx, 2, CF.tetragonal_variants(0.02, -0.005, 2), dt=0.005, cross_w=0.5, coupling=P.EIG_H,
                         elastic=P.ELAST_HETERO, ppt_scale=1.5, el_tol=1e-8, ny=ny, nz=nz)
    c, e = _fields(p, nx + ny + nz)
    o = oracle.OracleSim(p)
    o.set_fields(c, e)
    do = o.run(2)
    co, eo, eno, _ = o.get_fields()
    d, (cg, eg, eng, _) = _run(p, c, e, 2)
    assert list(d["el_iters"]) == list(do["el_iters"])
    # the gate of every FP64 path: 1e-10 on fields of order 1
    assert np.max(np.abs(cg - co)) <= 1e-10 and np.max(np.abs(eg - eo)) <= 1e-10
    assert np.max(np.abs(eng - eno)) <= 1e-10 * max(1.0, np.max(np.abs(eno)))
    # FP32 fields: a step rounds each value about 2 log2(N) + 10 times by 2^-24, with the local
    # solves in between amplifying by the modulus contrast (1.5): 64 roundings bound two steps
    q = p.copy()
    q.precision = P.PREC_F32
    _, (c32, e32, _, _) = _run(q, c, e, 2)
    bound = 64 * 2.0 ** -24
    assert np.linalg.norm(c32 - co) <= bound * np.linalg.norm(co)
    assert np.linalg.norm(e32 - eo) <= bound * np.linalg.norm(eo)


@pytest.mark.parametrize("nvar,numel,box", [(1, 2, (24, 16, 18)), (3, 2, (36, 12, 24)), (3, 3, (16, 54, 32)),
                                            (1, 2, (48, 36, 27)), (3, 2, (64, 8, 72)), (1, 3, (18, 24, 96))])
def test_kks_box_matches_oracle(oracle, nvar, numel, box):
    nx, ny, nz = box
    _, p, cons, phi = kks_case(nx, nvar, 4, numel_in=numel, ny=ny, nz=nz)
    rng = np.random.default_rng(nx * ny + nz)
    phi = np.clip(phi + 0.2 * rng.uniform(0, 1, phi.shape) * (rng.uniform(size=phi.shape) > 0.2), 0.0, 1.0)
    cons = cons + 0.01 * rng.uniform(-1, 1, cons.shape)
    o = oracle.OracleSim(p)
    o.set_fields(cons, phi)
    do = o.run(4)
    co, fo, eno, uo = o.get_fields()
    from meumapps_ss_b200.sim import Simulation
    with Simulation(p) as g:
        g.set_fields(cons, phi)
        d = g.run(4)
        cg, fg, eng, ug = g.get_fields(ustate=True)
    assert list(d["el_iters"]) == list(do["el_iters"])
    assert np.max(np.abs(cg - co)) <= 1e-10 and np.max(np.abs(fg - fo)) <= 1e-10
    assert np.max(np.abs(eng - eno)) <= 1e-9 * np.max(np.abs(eno))
    assert np.max(np.abs(ug - uo)) <= 1e-9 * np.max(np.abs(uo))
    for k in ("fint", "fch", "elen"):
        assert np.max(np.abs(d[k] - do[k])) <= 1e-9 * np.max(np.abs(do[k])), k


def test_kks_off_diagonal_gradient_tensor_matches_oracle(oracle):
    # gradient tensors with off-diagonal entries take the kappa-Laplacian through 3-D spectra
    _, p, cons, phi = kks_case(24, 3, 4, ny=16, nz=18 * 2)
    for v in range(3):
        g = p.grad_coeff[v][0]
        for i in (1, 3):
            p.grad_coeff[v][i] = 0.2 * g
        p.grad_coeff[v][5] = -0.1 * g
    rng = np.random.default_rng(5)
    phi = np.clip(phi + 0.2 * rng.uniform(0, 1, phi.shape) * (rng.uniform(size=phi.shape) > 0.2), 0.0, 1.0)
    o = oracle.OracleSim(p)
    o.set_fields(cons, phi)
    o.run(3)
    co, fo, _, _ = o.get_fields()
    _, (cg, fg, _, _) = _run(p, cons, phi, 3)
    assert np.max(np.abs(cg - co)) <= 1e-10 and np.max(np.abs(fg - fo)) <= 1e-10


def test_kks_fp32_one_variant_against_fp64():
    # the one-variant FP32 deck takes every fused path; bound as for the boxes above
    _, p, cons, phi = kks_case(36, 1, 4, ny=24, nz=32)
    rng = np.random.default_rng(9)
    phi = np.clip(phi + 0.2 * rng.uniform(0, 1, phi.shape), 0.0, 1.0)
    _, (c64, f64, _, _) = _run(p, cons, phi, 2)
    q = p.copy()
    q.precision = P.PREC_F32
    _, (c32, f32, _, _) = _run(q, cons, phi, 2)
    bound = 64 * 2.0 ** -24
    assert np.linalg.norm(c32 - c64) <= bound * np.linalg.norm(c64)
    assert np.linalg.norm(f32 - f64) <= bound * np.linalg.norm(f64)


def _landau_128(nvar, precision, kappa=1.0, n=128):
    eig = [[0.01] * 3] if nvar == 1 else CF.tetragonal_variants(0.02, -0.005, nvar)
    p = CF.landau_params(n, nvar, eig, dt=0.005, cross_w=0.5 if nvar > 1 else 0.0, precision=precision,
                         kappa_c=kappa, kappa_eta=kappa)
    return (p,) + _fields(p, 31)


@pytest.mark.parametrize("nvar,precision", [(2, P.PREC_F64), (3, P.PREC_F32), (4, P.PREC_F64)])
def test_default_plan_of_128_equals_plan_0(nvar, precision):
    # two plans of the same transforms: fields, loss and gradients differ by rounding alone, a few
    # units of a step's sums per step (64 units in the norms; the gradients' sums cancel, times 100).
    # Both schedules run the adjoint, each on its own order of the spectra.
    from meumapps_ss_b200.sim import Simulation
    p, c, e = _landau_128(nvar, precision)
    unit = 2.0 ** -24 if precision == P.PREC_F32 else 2.0 ** -53
    out = []
    for sched in (None, (0, 512, 16 if precision == P.PREC_F32 else 8)):
        with Simulation(p) as g:
            if sched:
                g.set_schedule(*sched)
            assert g.schedule[0] == (0 if sched else 2)
            g.set_fields(c, e)
            J, gr, ge = g.adjoint(3, 2, 0.9 * c, 0.5 * e)
        with Simulation(p) as g:
            if sched:
                g.set_schedule(*sched)
            g.set_fields(c, e)
            g.run(3)
            out.append((g.get_fields()[:2], J, gr, ge))
    (fa, Ja, ga, gea), (fb, Jb, gb, geb) = out
    for a, b in zip(fa, fb):
        assert np.linalg.norm(a - b) <= 64 * unit * np.linalg.norm(b)
    assert abs(Ja - Jb) <= 64 * unit * abs(Jb)
    assert np.linalg.norm(gea - geb) <= 64 * unit * np.linalg.norm(geb)
    for k in gb:
        assert abs(ga[k] - gb[k]) <= 6400 * unit * abs(gb[k]), k


def test_default_plane_threads_of_96_change_nothing():
    from meumapps_ss_b200.sim import Simulation
    p, c, e = _landau_128(1, P.PREC_F32, n=96)
    out = []
    for sched in (None, (0, 512, 16)):
        with Simulation(p) as g:
            if sched:
                g.set_schedule(*sched)
            assert g.schedule == (0, 512 if sched else 256, 16)
            g.set_fields(c, e)
            J, gr, ge = g.adjoint(3, 2, 0.9 * c, 0.5 * e)
            out.append((J, gr, ge))
    assert np.array_equal(out[0][2], out[1][2]) and out[0][0] == out[1][0] and out[0][1] == out[1][1]


@pytest.mark.parametrize("dims,precision", [((48, 36, 54), P.PREC_F64), ((64, 16, 32), P.PREC_F32)])
def test_chained_launches_repeat_bit_for_bit(dims, precision):
    # the step's kernels are placed before the one ahead of them ends; fixed-order sums and in-place
    # spectra make any read that came too early show as a difference between two runs
    nx, ny, nz = dims
    _, p, cons, phi = kks_case(nx, 3, 4, ny=ny, nz=nz)
    p.precision = precision
    rng = np.random.default_rng(3)
    phi = np.clip(phi + 0.2 * rng.uniform(0, 1, phi.shape), 0.0, 1.0)
    first = None
    for _ in range(6):
        _, (c, f, en, u) = _run(p, cons, phi, 4)
        if first is None:
            first = (c, f, en)
        assert all(np.array_equal(a, b) for a, b in zip(first, (c, f, en)))
