"""The passes that give a particle several lanes (few particles) against the ones that give it one:
the same particles alone, and together with enough others far away that the count takes the
general kernels.  Neighbour lists, densities, forces and the integrated state are the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FILL = np.stack(np.meshgrid(np.arange(28), np.arange(24), np.arange(30), indexing="ij"), -1).reshape(-1, 3) * 0.02
FILL = (FILL + np.array([0.5, -0.24, -0.29])).astype(np.float32)


def states():
    r = np.random.default_rng(3)
    def uniform(n, size):
        return np.array([-0.55, 0.0, 0.0]) + (r.random((n, 3)) - 0.5) * np.array(size)
    g = np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.02
    twins = uniform(130, (0.2, 0.2, 0.2))
    twins[60:100] = twins[0:40]   # coincident pairs
    odd = uniform(131, (0.2, 0.2, 0.2))
    odd[7] = np.nan
    odd[8, 2] = np.inf
    return {"one": uniform(1, (0.1,) * 3), "three": uniform(3, (0.02,) * 3), "lattice": g + (-0.7, -0.08, -0.08),
            "dense": uniform(2001, (0.24, 0.24, 0.24)),      # some with more than 64 members
            "crowd": uniform(1500, (0.07, 0.07, 0.07)),      # more than 1,024 candidates
            "twins": twins, "not_finite": odd, "walls": uniform(900, (1.2, 0.55, 0.6)) + (0.2, 0, 0),
            "last16": uniform(9728, (0.8, 0.5, 0.55)), "first8": uniform(9729, (0.8, 0.5, 0.55)),
            "last8": uniform(19456, (0.8, 0.5, 0.55))}


@pytest.mark.parametrize("name", ["one", "three", "lattice", "dense", "crowd", "twins", "not_finite", "walls",
                                  "last16", "first8", "last8"])
def test_same_bits_as_the_general_passes(gpu, name):
    import bubbles_gb300 as bb
    from bubbles_gb300 import scenes
    few = states()[name].astype(np.float32)
    n = len(few)
    assert len(FILL) > 19456
    vel = np.random.default_rng(5).normal(0, 0.3, (n, 3)).astype(np.float32)
    out = []
    for pos, v in ((few, vel), (np.concatenate([few, FILL]), np.concatenate([vel, np.zeros_like(FILL)]))):
        sc = scenes.base_scene("sph", 0.02, (2.4, 0.6, 0.7))
        with bb.Solver(sc, pos=pos, vel=v) as s:
            s.update_grid_distribution()
            s.compute_density(1)
            count, lists = s.neighbor_lists(min(200, 5 * n))
            s.advance_time_step(1e-4)
            rho, force = s.get(bb.FIELD_DENSITY), s.get(bb.FIELD_FORCE)
            x, u = s.download()
        out.append([np.asarray(a)[:n].copy() for a in (count, lists, rho, force, x, u)])
    for what, a, b in zip(("counts", "lists", "density", "force", "positions", "velocities"), *out):
        assert a.tobytes() == b.tobytes(), what


@pytest.mark.parametrize("name", ["one", "three", "lattice", "dense", "crowd", "twins", "walls", "last16", "first8",
                                  "last8"])
def test_same_bits_of_the_corrector(gpu, name):
    import bubbles_gb300 as bb
    from bubbles_gb300 import scenes
    few = states()[name].astype(np.float32)
    n = len(few)
    vel = np.random.default_rng(6).normal(0, 0.3, (n, 3)).astype(np.float32)
    out = []
    for pos, v in ((few, vel), (np.concatenate([few, FILL]), np.concatenate([vel, np.zeros_like(FILL)]))):
        sc = scenes.base_scene("pcisph", 0.02, (2.4, 0.6, 0.7))
        sc["pcisph_mode"] = "tolerance"
        sc["max_iterations"] = 4
        sc["max_density_error_ratio"] = 1e-12   # never met: both run all iterations
        with bb.Solver(sc, pos=pos, vel=v) as s:
            s.update_grid_distribution()
            s.advance_time_step(1e-4)
            fields = [s.get(f) for f in (bb.FIELD_DENSITY, bb.FIELD_PRESSURE, bb.FIELD_PRED_DENSITY,
                                         bb.FIELD_DENSITY_ERROR, bb.FIELD_PRESSURE_FORCE, bb.FIELD_FORCE)]
            fields += list(s.download())
        out.append([np.asarray(a)[:n].copy() for a in fields])
    for k, (a, b) in enumerate(zip(*out)):
        assert a.tobytes() == b.tobytes(), k
