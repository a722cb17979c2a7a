"""The three forms of the neighbour passes (several lanes a particle up to 19,456 particles, more loads in
flight up to 77,824, the general kernels past them) give the same bits: the states of
test_gpu_few_particles.py alone and beside enough far particles for the other two, and on both sides of the
line between them."""
import numpy as np
import pytest

from test_gpu_few_particles import states

pytestmark = pytest.mark.gpu

NAMES = ["one", "three", "lattice", "dense", "crowd", "twins", "not_finite", "walls", "last8"]
SIZE = (7.2, 0.6, 0.7)


def rest(n):
    g = np.stack(np.meshgrid(np.arange(150), np.arange(24), np.arange(30), indexing="ij"), -1).reshape(-1, 3)
    return (g[:n] * 0.02 + np.array([0.5, -0.24, -0.29])).astype(np.float32)


def runs(few, seed):
    n = len(few)
    vel = np.random.default_rng(seed).normal(0, 0.3, (n, 3)).astype(np.float32)
    for total in (n, 30000, 77824, 77825, 100000):
        r = rest(total - n)
        yield np.concatenate([few, r]), np.concatenate([vel, np.zeros_like(r)])


@pytest.mark.parametrize("name", NAMES)
def test_sph_substep(gpu, name):
    import bubbles_gb300 as bb
    from bubbles_gb300 import scenes
    few = states()[name].astype(np.float32)
    n, out = len(few), []
    for pos, vel in runs(few, 5):
        with bb.Solver(scenes.base_scene("sph", 0.02, SIZE), pos=pos, vel=vel) as s:
            s.update_grid_distribution()
            s.compute_density(1)
            got = list(s.neighbor_lists(200))
            s.advance_time_step(1e-4)
            got += [s.get(bb.FIELD_DENSITY), s.get(bb.FIELD_FORCE), *s.download()]
        out.append([np.asarray(a)[:n].copy() for a in got])
    for other in out[1:]:
        for what, a, b in zip(("counts", "lists", "density", "force", "positions", "velocities"), out[0], other):
            assert a.tobytes() == b.tobytes(), what


@pytest.mark.parametrize("name", [k for k in NAMES if k != "not_finite"])
def test_corrector(gpu, name):
    import bubbles_gb300 as bb
    from bubbles_gb300 import scenes
    few = states()[name].astype(np.float32)
    n, out = len(few), []
    for pos, vel in runs(few, 6):
        sc = scenes.base_scene("pcisph", 0.02, SIZE)
        # a tolerance never met: all of them run all iterations
        sc.update(pcisph_mode="tolerance", max_iterations=4, max_density_error_ratio=1e-12)
        with bb.Solver(sc, pos=pos, vel=vel) as s:
            s.update_grid_distribution()
            s.advance_time_step(1e-4)
            got = [s.get(f) for f in (bb.FIELD_DENSITY, bb.FIELD_PRESSURE, bb.FIELD_PRED_DENSITY,
                                      bb.FIELD_DENSITY_ERROR, bb.FIELD_PRESSURE_FORCE, bb.FIELD_FORCE)]
            got += list(s.download())
        out.append([np.asarray(a)[:n].copy() for a in got])
    for other in out[1:]:
        for k, (a, b) in enumerate(zip(out[0], other)):
            assert a.tobytes() == b.tobytes(), k
