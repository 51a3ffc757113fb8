"""Non-finite values in a disk without a v_z: the step that leaves the v_z planes
out gives the v_z that the five-plane step would, NaN where 0 times an infinity
or a NaN enters it.  The bad cell is in the outer ghost annulus, so that the
first step's CFL minimum is finite; the state after the step against the
oracle's C restatement, NaN for NaN and every other value bit for bit."""
import os

import numpy as np
import pytest

import oracle
from disco2_b200 import configs, lib

pytestmark = pytest.mark.gpu

NAN, INF = float("nan"), float("inf")
BAD = [{0: NAN}, {0: INF}, {1: NAN}, {1: INF}, {2: NAN}, {2: INF}, {2: -INF}, {3: INF}, {0: 1e300, 2: 1e300}]


@pytest.mark.parametrize("over", [{}, {"RiemannSolver": 1}, {"BoundTypeR": 1}], ids=str)
@pytest.mark.parametrize("bad", BAD, ids=str)
def test_nonfinite_cell(bad, over, tmp_path):
    p = configs.gresho(6, NP_CONST=24, w_numeric_type=0, **over)
    par = configs.write_parfile(p, os.path.join(str(tmp_path), "g.par"))
    st, _, _ = oracle.run(par, 0, impl="port")
    st.prim[:, 4] = 0.0
    for q, v in bad.items():
        st.prim[-7, q] = v
    want, _, _ = oracle.run(par, 1, impl="port", load=st)
    ctx = lib.Context(lib.Sim(p))
    ctx.init_state(0)
    ctx.set_state(0, st.prim, st.tiph, st.dphi)
    ctx.step(1)
    got = ctx.get_state(0)
    ctx.close()
    for k in ("prim", "cons", "tiph", "dphi"):
        assert np.array_equal(got[k], getattr(want, k), equal_nan=True), k
