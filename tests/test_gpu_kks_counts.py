"""The KKS driving force with every variant count that has compiled-in registers, against the oracle."""
import numpy as np
import pytest

from meumapps_ss_b200 import configs as CF
from meumapps_ss_b200 import params as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("numel", [1, 2])
@pytest.mark.parametrize("nvar", range(1, 17))
def test_variant_count_matches_oracle(oracle, nvar, numel):
    from meumapps_ss_b200.sim import Simulation
    deck = P.parse_input_txt(CF.kks_input_txt(16, nvar, 10, numel_in=numel + 1, ny=6, nz=9))
    p = P.kks_params(deck, sym_var=CF.tetrahedral_rotations())
    # the deck reader orients 1, 3 and 12 variants; here every count gets gradient energy and a strain
    # (without gradients an absent variant stays at zero but for rounding, whose sign n_tilda would count)
    eig = CF.tetragonal_variants(0.02, -0.005, nvar)
    for v in range(nvar):
        for i in range(9):
            p.grad_coeff[v][i] = 5.0e8 if i % 4 == 0 else 0.0
        for i in range(6):
            p.trans_ppt[v][i] = eig[v][i] if i < 3 else 0.0
    cons, phi = P.init_fields(deck)
    rng = np.random.default_rng(100 * numel + nvar)
    # every variant present, and absent in a fifth of the voxels (the n_tilda projection counts those above 0)
    phi = np.clip(phi + 0.4 / nvar * rng.uniform(0.01, 1, phi.shape) * (rng.uniform(size=phi.shape) > 0.2), 0.0, 1.0)
    cons = cons + 0.01 * rng.uniform(-1, 1, cons.shape)
    o = oracle.OracleSim(p)
    o.set_fields(cons, phi)
    do = o.run(2)
    co, fo, eno, _ = o.get_fields()
    with Simulation(p) as g:
        g.set_fields(cons, phi)
        d = g.run(2)
        cg, fg, eng, _ = g.get_fields()
    assert list(d["el_iters"]) == list(do["el_iters"])
    assert np.max(np.abs(cg - co)) <= 1e-10 and np.max(np.abs(fg - fo)) <= 1e-10
    assert np.max(np.abs(eng - eno)) <= 1e-9 * np.max(np.abs(eno))
    for k in ("fint", "fch", "fw", "elen"):
        assert np.max(np.abs(d[k] - do[k])) <= 1e-9 * np.max(np.abs(do[k])), k
