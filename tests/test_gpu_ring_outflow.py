"""The rigid ring mean and the outflow boundary at the sizes where their
kernels change path, against the oracle's C restatement run on the host: the
Gresho vortex reaches no transcendental, so the states are equal bit for bit.

Ring means are added 128 cells at a time, loaded 32 by 32; outflow boundary
cells take 8 faces at a time, and a disk of three annuli chains all
three passes.
"""
import os

import numpy as np
import pytest

import oracle
from disco2_b200 import configs, lib

pytestmark = pytest.mark.gpu

RINGS = [{"NP_CONST": n} for n in (2, 31, 32, 33, 65, 127, 128, 129, 257)]
OUT = {"BoundTypeR": 1}
OUTFLOW = [
    {"num_r": 1, "NP_CONST": 7, **OUT},                      # three annuli
    {"num_r": 1, "NP_CONST": 40, "NoInnerBC": 1, **OUT},     # three, no inner boundary
    {"num_r": 2, "NP_CONST": 33, **OUT},                     # NR-3 is annulus 1
    {"num_r": 1, "R_Min": 0.5, "R_Max": 0.9, "aspect": 0.45, **OUT},   # three: 2, 16, 30 cells
    {"num_r": 4, "R_Min": 0.15, "R_Max": 0.55, "aspect": 0.1, **OUT},  # 6 cells face 69
    {"num_r": 12, "ng": 2, **OUT},
]


def _check(over, tmp_path):
    over = dict(over)
    p = configs.gresho(over.pop("num_r", 4), **over)
    sim = lib.Sim(p)
    ctx = lib.Context(sim)
    ctx.init_state(0)
    ctx.step(3)
    got = ctx.get_state(0)
    ctx.close()
    par = configs.write_parfile(p, os.path.join(str(tmp_path), "g.par"))
    want, _, _ = oracle.run(par, 3, impl="port")
    for k in ("prim", "cons", "tiph", "dphi"):
        assert np.array_equal(got[k], getattr(want, k)), k


@pytest.mark.parametrize("over", RINGS, ids=str)
def test_rigid_ring_mean(over, tmp_path):
    _check(over, tmp_path)


@pytest.mark.parametrize("over", OUTFLOW, ids=str)
def test_outflow_boundary(over, tmp_path):
    _check(over, tmp_path)
