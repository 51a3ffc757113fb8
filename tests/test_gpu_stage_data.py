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


def _gresho(vz):
    sim = lib.Sim(configs.gresho(9))
    st = sim.initial_state()
    prim = st["prim"].copy()
    prim[:, 4] = vz * np.random.default_rng(2).uniform(0.5, 1.0, len(prim))
    return sim, prim, st


KEYS = ("grad", "gradp", "RKcons")


def test_stage_data_after_steps_with_and_without_vz():
    """After plain steps the arrays are the last substep's, also of a context
    that held a v_z before: the v_z slopes of a disk without one are 0."""
    sim, moving, st = _gresho(0.02)
    _, still, _ = _gresho(0.0)
    ctx = lib.Context(sim)
    ctx.init_state(0)
    want = {}
    for name, prim in (("moving", moving), ("still", still), ("moving", moving), ("still", still)):
        for fused in (False, True):
            ctx.set_fused(fused)
            ctx.set_state(0, prim, st["tiph"], st["dphi"])
            ctx.set_time(0, 0.0)
            ctx.step(2)
            got = ctx.stage_data(0)
            for k in KEYS:
                if name == "still":
                    assert np.all(got[k][:, 4] == 0.0), k
                else:
                    assert np.any(got[k][:, 4] != 0.0), k
                assert np.array_equal(got[k], want.setdefault((name, k), got[k])), (name, fused, k)
    ctx.close()


def test_stage_after_steps_without_vz():
    """dgpu_stage on a state with a v_z, the steps before it without one."""
    sim, moving, st = _gresho(0.02)
    _, still, _ = _gresho(0.0)
    out = []
    for steps in (0, 2):
        ctx = lib.Context(sim)
        ctx.init_state(0)
        ctx.set_state(0, still, st["tiph"], st["dphi"])
        ctx.step(steps)
        ctx.set_state(0, moving, st["tiph"], st["dphi"])
        ctx.set_time(0, 0.0)
        ctx.stage(1)
        out.append(ctx.stage_data(0))
        ctx.close()
    for k in KEYS:
        assert np.any(out[0][k][:, 4] != 0.0) and np.array_equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("make", [configs.gresho, configs.kepler_ring], ids=lambda f: f.__name__)
def test_wiph_after_face_list(make):
    """The face list of a newly set state brings wiph with it, on a rigidly
    rotating mesh too (the ring means of that state)."""
    sim = lib.Sim(make(9))
    st = sim.initial_state()
    prim = st["prim"].copy()
    prim[:, 3] *= 1.5
    ctx = lib.Context(sim)
    ctx.init_state(0)
    ctx.step(1)
    ctx.set_state(0, prim, st["tiph"], st["dphi"])
    ctx.face_list(0)
    got = ctx.stage_data(0)["wiph"]
    ctx.stage(0)
    want = ctx.stage_data(0)["wiph"]
    ctx.close()
    assert np.array_equal(got, want)
