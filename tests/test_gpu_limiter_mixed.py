"""The r-slope limiter of cells whose face slopes differ by up to 300 decades:
there a clipped running slope times an opposed one underflows while the mean's
product does not.  The slopes against the oracle's C restatement bit for bit;
the reverse of the limiter against the forward-mode tangent (the bar of the
gradient tests, 1e-9 relative)."""
import os

import numpy as np
import pytest

import oracle
from disco2_b200 import configs, lib

pytestmark = pytest.mark.gpu

SIZES = np.array([0.0, 1e-170, -1e-170, 2e-170, -3e-170, 1e-100, -1e-100, 1e-20])


@pytest.mark.parametrize("over", [{"num_r": 5, "NP_CONST": 19}, {"num_r": 8, "R_Min": 0.2}, {"num_r": 9, "PLM": 1.0}],
                         ids=str)
def test_limiter_of_mixed_slopes(over, tmp_path):
    over = dict(over)
    p = configs.gresho(over.pop("num_r"), **over)
    par = configs.write_parfile(p, os.path.join(str(tmp_path), "g.par"))
    st, _, _ = oracle.run(par, 0, impl="port")
    ctx = lib.Context(lib.Sim(p))
    ctx.init_state(0)
    for seed in range(6):
        rng = np.random.default_rng(seed)
        st.prim[:, 2] = rng.choice(SIZES, st.prim.shape[0])
        st.prim[:, 4] = rng.choice(SIZES, st.prim.shape[0])
        want = oracle.stage(par, 1, impl="port", load=st)
        ctx.set_state(0, st.prim, st.tiph, st.dphi)
        ctx.stage(1)
        assert np.array_equal(ctx.stage_data(0)["grad"], want.ext["grad"]), seed
    ctx.close()


def test_reverse_of_mixed_slopes():
    sim = lib.Sim(configs.kepler_ring(7, NP_CONST=63, CFL=0.2))
    ctx = lib.Context(sim)
    ctx.init_state(0)
    st = ctx.get_state(0)
    rng = np.random.default_rng(3)
    prim = st["prim"]
    prim[:, 0] *= 1.0 + 0.05 * rng.uniform(-1.0, 1.0, len(prim))
    prim[:, 2] = rng.choice(SIZES, len(prim))
    d = np.zeros_like(prim)
    d[:, 2] = rng.uniform(-1.0, 1.0, len(prim))
    gm = ctx.gravmass(0)

    def reset():
        ctx.set_state(0, prim, st["tiph"], st["dphi"])
        ctx.set_gravmass(0, gm)
        ctx.set_time(0, 0.0)

    reset()
    g = ctx.adjoint(2, 1, ckpt_every=2, weights=(0.0, 1.0))
    reset()
    _, dJ = ctx.tangent(2, 1, dprim=d)
    ctx.close()
    along = float((g["dprim"] * d).sum())
    scale = float(np.abs(g["dprim"] * d).sum())
    assert abs(along - dJ[1]) <= 1e-9 * scale


def test_limiter_with_negative_plm(tmp_path):
    """A PLM below zero turns the slope's sign at every face that clips it."""
    p = configs.gresho(8, R_Min=0.2, PLM=-0.7)
    par = configs.write_parfile(p, os.path.join(str(tmp_path), "g.par"))
    st, _, _ = oracle.run(par, 0, impl="port")
    st.prim += 0.05 * np.random.default_rng(1).uniform(-1.0, 1.0, st.prim.shape)
    want = oracle.stage(par, 1, impl="port", load=st)
    ctx = lib.Context(lib.Sim(p))
    ctx.init_state(0)
    ctx.set_state(0, st.prim, st.tiph, st.dphi)
    ctx.stage(1)
    assert np.array_equal(ctx.stage_data(0)["grad"], want.ext["grad"])
    ctx.close()
