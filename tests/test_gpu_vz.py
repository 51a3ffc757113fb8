"""Disks with and without a v_z: the step leaves out the v_z planes of a
context whose uploads held none, and takes them again as soon as one does.
Against the oracle's C restatement from the same states; the Gresho vortex
(no transcendental) bit for bit."""
import os

import numpy as np
import pytest

import oracle
from conftest import max_rel
from disco2_b200 import configs, lib

pytestmark = pytest.mark.gpu

KEYS = ("prim", "cons", "tiph", "dphi")


def _start(par, vz):
    st, _, _ = oracle.run(par, 0, impl="port")
    rng = np.random.default_rng(11)
    st.prim[:, 2] = 0.01 * rng.uniform(-1.0, 1.0, st.prim.shape[0])
    st.prim[:, 4] = vz * rng.uniform(-1.0, 1.0, st.prim.shape[0])
    return st


def _gresho(tmp_path, num_r, **over):
    p = configs.gresho(num_r, **over)
    return p, configs.write_parfile(p, os.path.join(str(tmp_path), f"g{num_r}.par"))


@pytest.mark.parametrize("over", [{"NP_CONST": 33}, {"RiemannSolver": 1}, {"BoundTypeR": 1}], ids=str)
def test_one_context_with_and_without_vz(over, tmp_path):
    p, par = _gresho(tmp_path, 9, **over)
    ctx = lib.Context(lib.Sim(p))
    ctx.init_state(0)
    for vz in (0.0, 0.02, 0.0, 1e-200, 0.0):
        st = _start(par, vz)
        want, _, _ = oracle.run(par, 3, impl="port", load=st)
        ctx.set_state(0, st.prim, st.tiph, st.dphi)
        ctx.set_time(0, 0.0)
        ctx.step(3)
        got = ctx.get_state(0)
        for k in KEYS:
            assert np.array_equal(got[k], getattr(want, k)), (vz, k)
    ctx.close()


def test_one_disk_of_two_has_vz(tmp_path):
    ps = [_gresho(tmp_path, n) for n in (12, 15)]
    ctx = lib.Context([lib.Sim(p) for p, _ in ps])
    for vzs in ((0.0, 0.02), (0.01, 0.0), (0.0, 0.0)):
        sts = [_start(par, vz) for (_, par), vz in zip(ps, vzs)]
        for k, st in enumerate(sts):
            ctx.set_state(k, st.prim, st.tiph, st.dphi)
            ctx.set_time(k, 0.0)
        ctx.step(2)
        for k, st in enumerate(sts):
            want, _, _ = oracle.run(ps[k][1], 2, impl="port", load=st)
            got = ctx.get_state(k)
            for q in KEYS:
                assert np.array_equal(got[q], getattr(want, q)), (vzs, k, q)
    ctx.close()


def test_vertical_gravity_makes_vz(tmp_path):
    """A single layer off the midplane: v_z grows from 0 (the torus' bar of a
    few steps, 1e-12)."""
    p = configs.torus_2d(16, Z_Min=-0.5, Z_Max=1.0)
    par = configs.write_parfile(p, os.path.join(str(tmp_path), "t.par"))
    ctx = lib.Context(lib.Sim(p))
    ctx.init_state(0)
    ctx.step(3)
    got = ctx.get_state(0)
    ctx.close()
    want, _, _ = oracle.run(par, 3, impl="port")
    assert np.abs(want.prim[:, 4]).max() > 0.0
    for k in KEYS:
        assert max_rel(got[k], getattr(want, k)) <= 1e-12, k
