"""The stage arrays (stage_data) outside the plain case that the parity tests
cover."""
import numpy as np
import pytest

from disco2_b200 import configs, lib

pytestmark = pytest.mark.gpu


def test_wiph_of_every_layer():
    """A 3-D disk on the Keplerian mesh: the layers' annuli move alike."""
    sim = lib.Sim(configs.torus_3d(num_r=16, num_z=8, w_numeric_type=3))
    ctx = lib.Context(sim)
    ctx.init_state(0)
    ctx.step(1)
    w = ctx.stage_data(0)["wiph"]
    ctx.close()
    layer = int(sum(sim.grid()[0]))
    w = w.reshape(-1, layer)
    assert w.shape[0] == 12 and np.all(w[0] != 0.0)
    assert np.array_equal(w, np.broadcast_to(w[0], w.shape))
