"""The r-slope limiter where the products of opposed slopes underflow, and
where face slopes are exactly zero: there the one walk over a cell's faces does
not decide and the reference's face-by-face loop runs.  Against the oracle's
C restatement from the same state, bit for bit (Gresho: no transcendental)."""
import os

import numpy as np
import pytest

import oracle
from disco2_b200 import configs, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-3, 1e-150, 1e-165, 1e-300, 0.0])
@pytest.mark.parametrize("over", [{"num_r": 5, "NP_CONST": 19}, {"num_r": 8, "R_Min": 0.2}], ids=str)
def test_limiter_of_tiny_slopes(over, scale, tmp_path):
    over = dict(over)
    p = configs.gresho(over.pop("num_r"), **over)
    par = configs.write_parfile(p, os.path.join(str(tmp_path), "g.par"))
    st, _, _ = oracle.run(par, 0, impl="port")
    rng = np.random.default_rng(5)
    vr = scale * rng.integers(-2, 3, st.prim.shape[0])  # signs of both kinds, and zeros
    st.prim[:, 2] = vr
    sim = lib.Sim(p)
    ctx = lib.Context(sim)
    ctx.init_state(0)
    ctx.set_state(0, st.prim, st.tiph, st.dphi)
    for phase in (1, 9):
        want = oracle.stage(par, phase, impl="port", load=st)
        ctx.set_state(0, st.prim, st.tiph, st.dphi)
        ctx.stage(phase)
        assert np.array_equal(ctx.stage_data(0)["grad"], want.ext["grad"]), phase
    ctx.close()
