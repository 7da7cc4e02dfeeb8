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
