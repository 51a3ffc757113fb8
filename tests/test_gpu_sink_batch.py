"""Sink accretion (Mdot, Macc) of disks that share a context: the sums of one
disk take in no cell of another, where blocks of 256 cells hold the end of one
disk and the start of the next, or several whole disks.  Against the same disk
alone: the same non-negative terms, at most 300 of them, grouped otherwise, so
equal within 300 rounding errors (3.4e-14 relative)."""
import numpy as np
import pytest

from disco2_b200 import configs, lib

pytestmark = pytest.mark.gpu


def _run(ps, nsteps=3):
    ctx = lib.Context([lib.Sim(p) for p in ps])
    for k in range(len(ps)):
        ctx.init_state(k)
    ctx.step(nsteps)
    out = [ctx.gravmass(k) for k in range(len(ps))]
    ctx.close()
    return out


@pytest.mark.parametrize("disks", [
    [128, 128],              # 262 cells each: block 1 ends disk 0 and starts disk 1
    [128, 32, 40, 36, 131],  # 262 + 70 + 86 + 78 + 268: five disks in block 1
    [125, 125, 0],           # 256 cells each: boundaries on blocks' edges; a disk without sink
], ids=str)
def test_accretion_of_batched_disks(disks):
    ps = [configs.sstest(n) if n else configs.kepler_ring(24) for n in disks]
    got = _run(ps)
    for k, p in enumerate(ps):
        want = _run([p])[0]
        if disks[k]:
            assert want[0, 4] > 0.0 and want[0, 5] > 0.0
        for q in (4, 5):  # Mdot, Macc
            assert np.all(np.abs(got[k][:, q] - want[:, q]) <= 3.4e-14 * want[:, q]), (k, q, got[k][:, q], want[:, q])
