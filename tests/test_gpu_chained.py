"""Steps whose kernels are placed before the one ahead of them ends: fixed-order sums and in-place
spectra make any read that came too early show as a difference between two runs.  Every precision
and model that takes the elastic rows, the one-axis derivatives and the fused z updates."""
import numpy as np
import pytest

from meumapps_ss_b200 import configs as CF
from meumapps_ss_b200 import params as P

pytestmark = pytest.mark.gpu

ROWS = ("el_iters", "fint", "fch", "fw", "elen", "cmin", "cmax", "phimax", "solid_now", "cavg")


def _kks(precision, nvar, dims):
    deck = P.parse_input_txt(CF.kks_input_txt(dims[0], nvar, 10, ny=dims[1], nz=dims[2]))
    p = P.kks_params(deck, precision=precision, sym_var=CF.tetrahedral_rotations())
    cons, phi = P.init_fields(deck)
    rng = np.random.default_rng(3)
    return p, cons, np.clip(phi + 0.2 * rng.uniform(0, 1, phi.shape), 0.0, 1.0)


def _hetero(precision, nvar, dims):
    p = CF.landau_params(dims[0], nvar, CF.tetragonal_variants(0.02, -0.005, nvar), dt=0.005, cross_w=0.5,
                         coupling=P.EIG_H, elastic=P.ELAST_HETERO, ppt_scale=1.5, el_tol=1e-8, precision=precision,
                         ny=dims[1], nz=dims[2])
    rng = np.random.default_rng(5)
    s = (p.nz, p.ny, p.nx)
    return p, 0.8 + 0.05 * rng.uniform(-1, 1, (1,) + s), 0.5 * rng.uniform(-1, 1, (nvar,) + s)


@pytest.mark.parametrize("make,precision,nvar,dims", [
    (_kks, P.PREC_F32, 1, (48, 36, 54)), (_kks, P.PREC_F32, 1, (64, 16, 32)), (_kks, P.PREC_F64, 12, (54, 24, 36)),
    (_hetero, P.PREC_F32, 3, (54, 36, 72)), (_hetero, P.PREC_F64, 3, (54, 36, 72)), (_hetero, P.PREC_F32, 4, (128, 32, 16)),
    (_hetero, P.PREC_F64, 2, (96, 24, 27)), (_hetero, P.PREC_F64, 12, (512, 9, 8))])
def test_runs_repeat_bit_for_bit(make, precision, nvar, dims):
    from meumapps_ss_b200.sim import Simulation
    p, c, e = make(precision, nvar, dims)
    first = None
    for _ in range(6):
        with Simulation(p) as g:
            g.set_fields(c, e)
            d = g.run(4)
            f = g.get_fields(ustate=True)
        if first is None:
            first = (d, f)
            assert all(np.all(np.isfinite(a)) for a in f)
        assert all(np.array_equal(a, b) for a, b in zip(f, first[1]))
        assert all(np.array_equal(d[k], first[0][k]) for k in ROWS)
