"""Dilts' test of scattered particles, told by a thread each, beside dense ones, told by a warp each, at
every number of particles a block takes: against the oracle.  And the cost of scattered particles."""
import time

import numpy as np
import pytest

import bubbles_gb300 as bb
from bubbles_gb300 import scenes
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# a block takes 4 particles up to 38,912, then 8, 16 (from 77,825) and 32 (from 155,649)
@pytest.mark.parametrize("n", [1, 5, 2003, 38913, 77830, 155700])
def test_scattered_and_dense_particles(gpu, n):
    r = np.random.default_rng(n)
    side = np.array([2.4, 1.2, 1.6])
    pos = (r.random((n, 3)) - 0.5) * (side - 0.06)
    m = min(n // 2, 900)
    clump = np.stack(np.meshgrid(*[np.arange(10)] * 3, indexing="ij"), -1).reshape(-1, 3)[:m] * 0.012
    pos[:m] = clump + r.uniform(-0.002, 0.002, (m, 3))
    if n > 100:
        pos[-40:-20] = pos[-60:-40]                         # pairs in one place: each holds the other's points
        pos[-20:] = pos[-60:-40] + [0.0, 0.0, 0.017]        # above it: the first point only
    pos = pos[r.permutation(n)].astype(np.float32)
    sc = scenes.base_scene("pcisph", 0.02, tuple(side))
    o = O.OracleSim(sc, pos)
    o.update_grid_distribution()
    want = o.dilts()
    o.close()
    with bb.Solver(sc, pos=pos) as s:
        s.update_grid_distribution()
        got = s.boundary_test("dilts")
        levels, queued, accepted = s.lnm_boundary_geometric(0.02, "dilts")
    assert np.array_equal(got, want)
    assert accepted == int((levels == 2).sum()) <= queued
    assert np.array_equal(want[levels == 2], np.ones(accepted, want.dtype))
    if n > 2000:
        assert 0 < want.sum() < n


def test_cost_of_scattered_particles(gpu):
    """A scattered particle has the same candidates to look at in Dilts' test as in Xiaowei's, and one
    point against one weight each: at most 3 times as long here, for what a block starts with."""
    g = np.stack(np.meshgrid(*[np.arange(60)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.03
    pos = (g - g.mean(0) + np.random.default_rng(1).uniform(-0.001, 0.001, g.shape)).astype(np.float32)
    took = []
    with bb.Solver(scenes.base_scene("pcisph", 0.01, (2.0,) * 3), pos=pos) as s:
        s.update_grid_distribution()
        s.compute_density(0)
        for test in ("xiaowei", "dilts"):
            best = float("inf")
            for _ in range(10):
                t = time.perf_counter()
                for _ in range(10):
                    s.boundary_test(test, 0.01)
                best = min(best, time.perf_counter() - t)
            took.append(best)
    assert took[1] <= 3.0 * took[0], took
