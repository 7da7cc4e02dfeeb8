"""Schedules that a caller names run as named; defaults and saved files keep their meaning."""
import os
import subprocess
import sys

import numpy as np
import pytest

from helpers import kks_case
from meumapps_ss_b200 import configs as CF
from meumapps_ss_b200 import params as P

pytestmark = pytest.mark.gpu

ROOT = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..")


def test_generic_plan_that_is_set_runs_in_every_pass():
    # FP64 columns of 128: a handle that sets nothing takes radix 16 for the inverse.  (0, 0, 1) and
    # (0, 0, 2) are both radix 8, one line's arithmetic, and differ in the columns per block alone.
    from meumapps_ss_b200.sim import Simulation
    _, p, cons, phi = kks_case(32, 1, 4, ny=128, nz=16)
    rng = np.random.default_rng(2)
    phi = np.clip(phi + 0.2 * rng.uniform(0, 1, phi.shape), 0.0, 1.0)
    out = []
    for ct in (1, 2):
        with Simulation(p) as g:
            assert g.schedule == (0, 0, 1)
            g.set_schedule(0, 0, ct)
            assert g.schedule == (0, 0, ct)
            g.set_fields(cons, phi)
            g.run(2)
            out.append(g.get_fields(ustate=True))
    assert all(np.array_equal(a, b) for a, b in zip(*out))


def test_saved_schedule_without_a_tile_is_the_wide_tile(tmp_path):
    saved = tmp_path / "tuned.txt"
    saved.write_text("f32 32 2 1 1 0 512 0 0.02\nf64 32 2 1 1 0 512 0 0.02\n")
    code = ("from helpers import active_landau\n"
            "from meumapps_ss_b200 import params as P\n"
            "from meumapps_ss_b200.sim import Simulation\n"
            "for prec, tm in ((P.PREC_F32, 16), (P.PREC_F64, 8)):\n"
            "    p, c, e = active_landau(32, 2, precision=prec)\n"
            "    p.flags |= P.FLAG_AUTOTUNE\n"
            "    with Simulation(p) as g:\n"
            "        assert g.schedule == (0, 512, tm), g.schedule\n"
            "        g.set_fields(c, e)\n"
            "        g.run(1)\n")
    env = dict(os.environ, MEU_AUTOTUNE_CACHE=str(saved),
               PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests"), os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", code], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("n,nvar,precision,tile", [(32, 2, P.PREC_F64, 8), (32, 3, P.PREC_F64, 4), (48, 2, P.PREC_F64, 8),
                                                   (48, 3, P.PREC_F64, 4), (64, 4, P.PREC_F64, 8),
                                                   (32, 1, P.PREC_F32, 16), (32, 2, P.PREC_F32, 8)])
def test_default_column_tile(n, nvar, precision, tile):
    # the narrow tile only where a single grid gains more from it than an ensemble of such grids loses
    from meumapps_ss_b200.sim import Ensemble, Simulation
    eig = [[0.01] * 3] if nvar == 1 else CF.tetragonal_variants(0.02, -0.005, nvar)
    p = CF.landau_params(n, nvar, eig, precision=precision)
    with Simulation(p) as g:
        assert g.schedule == (0, 512, tile)
    assert Ensemble([p, p]).schedule(1)[:3] == (0, 512, tile)


@pytest.mark.parametrize("nz,pv,fused_z", [(32, 0, True), (64, 0, True), (512, 0, True), (64, 2, False), (128, 0, False),
                                           (16, 0, False)])
def test_fp32_variants_keep_the_rounding_of_their_z_plan(nz, pv, fused_z):
    # FP32 decks of several variants run the fused z kernel only where its radix plan is the one that
    # the separate passes would run; the plan that a caller sets is kept either way
    from meumapps_ss_b200.sim import Simulation
    _, p, cons, phi = kks_case(16, 3, 4, ny=8, nz=nz)
    rng = np.random.default_rng(nz)
    # every variant present everywhere: n_tilda counts signs that rounding does not decide
    phi = np.clip(phi + rng.uniform(0.1, 0.3, phi.shape), 0.0, 1.0)
    out = {}
    for prec in (P.PREC_F64, P.PREC_F32):
        q = p.copy()
        q.precision = prec
        with Simulation(q) as g:
            if pv:
                g.set_schedule(pv, 0, 1)
            g.set_fields(cons, phi)
            g.timing(True)
            g.run(2)
            names = set(g.timing_report())
            out[prec] = g.get_fields()
        assert ("el_z" in names) == (fused_z or prec == P.PREC_F64), names
    # FP32 fields: 64 roundings bound two steps
    for a, b in zip(out[P.PREC_F32][:2], out[P.PREC_F64][:2]):
        assert np.linalg.norm(a - b) <= 64 * 2.0 ** -24 * np.linalg.norm(b)
