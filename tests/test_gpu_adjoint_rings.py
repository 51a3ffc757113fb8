"""The reverse of the phi slopes at ring sizes around its blocks: rings of two
cells (the neighbour on both sides is one cell), and rings that end in, fill
and span the blocks of 252 cells.  The gradient along a random direction
against the forward-mode tangent, which shares none of the reverse kernels
(the bar of the gradient tests, 1e-9 relative)."""
import numpy as np
import pytest

from disco2_b200 import configs, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 63, 126, 251, 252, 253, 509])
def test_gradient_against_tangent(n):
    sim = lib.Sim(configs.kepler_ring(7, NP_CONST=n, CFL=0.2))
    ctx = lib.Context(sim)
    ctx.init_state(0)
    st = ctx.get_state(0)
    rng = np.random.default_rng(n)
    prim = st["prim"]
    prim[:, 0] *= 1.0 + 0.05 * rng.uniform(-1.0, 1.0, len(prim))
    prim[:, 2] += 0.02 * rng.uniform(-1.0, 1.0, len(prim))
    d = prim * rng.uniform(-1.0, 1.0, prim.shape)
    gm = ctx.gravmass(0)

    def reset():
        ctx.set_state(0, prim, st["tiph"], st["dphi"])
        ctx.set_gravmass(0, gm)
        ctx.set_time(0, 0.0)

    reset()
    g = ctx.adjoint(4, 1, ckpt_every=2, weights=(0.0, 1.0))
    reset()
    _, dJ = ctx.tangent(4, 1, dprim=d)
    ctx.close()
    along = float((g["dprim"] * d).sum())
    scale = float(np.abs(g["dprim"] * d).sum())
    assert abs(along - dJ[1]) <= 1e-9 * scale
