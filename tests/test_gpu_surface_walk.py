"""The particle field's walk where its lists and loops end: scattered particles (columns taken at once),
dense ones (lists summed up between columns), cells of more particles than a list, radii of less than a
cell and of several, and node counts that leave warps part empty; against the oracle, bit for bit.
And the cost of the fields whose nodes sum most of their candidates."""
import time

import numpy as np
import pytest

import bubbles_gb300 as bb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def lattice(side, step):
    return np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3) * step


def states():
    r = np.random.default_rng(11)
    scattered = r.random((400, 3)) * 0.4
    dense = lattice(13, 0.0125) + r.uniform(-0.002, 0.002, (13 ** 3, 3))
    clump = np.concatenate([0.1 + 0.03 * r.random((300, 3)), r.random((200, 3)) * 0.3])   # cells past a list
    few = r.random((5, 3)) * np.array([0.3, 0.05, 0.02])
    return {"scattered": scattered, "lattice": lattice(9, 0.02) + r.uniform(-0.004, 0.004, (729, 3)), "dense": dense,
            "clump": clump, "few": few}


@pytest.mark.parametrize("name", ["scattered", "lattice", "dense", "clump", "few"])
@pytest.mark.parametrize("kernel,mc", [(0.04, 0.013), (0.1, 0.017), (0.012, 0.02)])
def test_fields_match_the_oracle(gpu, name, kernel, mc):
    pos = states()[name].astype(np.float32)
    sc = bb.surface_scene(pos, 0.02)
    o = O.OracleSim(sc, pos)
    o.update_grid_distribution()
    o.compute_density(0)
    rho = o.get(O.DENSITY)
    want = [o.particle_sdf(m, kernel, mc) for m in (0, 1)]
    o.close()
    with bb.Solver(sc, pos=pos) as s:
        s.update_grid_distribution()
        s.set(bb.FIELD_DENSITY, rho)
        for m in (0, 1):
            nodes, org, sp, vals = s.particle_sdf(m, kernel, mc)
            assert np.array_equal(nodes, want[m][0])
            assert vals.astype(np.float32).tobytes() == want[m][3].tobytes(), m


@pytest.mark.parametrize("step", [1.0, 0.8])
def test_cost_of_wide_radii_and_of_the_sph_field(gpu, step):
    """The walk over the 27 cells is the same for every radius; a weight costs about two tests, and a
    node that sums all its candidates instead of an eighth of them takes (1 + 2) / (1 + 2 / 8) = 2.4
    times as long.  At most 3 times here."""
    s = 0.01
    g = lattice(30, s * step)
    pos = (g - g.mean(0) + np.random.default_rng(1).uniform(-0.1, 0.1, g.shape) * s).astype(np.float32)
    took = []
    with bb.Solver(bb.surface_scene(pos, s), pos=pos) as q:
        q.update_grid_distribution()
        q.compute_density(0)
        for method, radius in (("zhu", 2 * s), ("zhu", 4 * s), ("sph", 2 * s)):
            best = float("inf")
            for _ in range(10):
                t = time.perf_counter()
                for _ in range(10):
                    q.particle_sdf(method, radius, s)
                best = min(best, time.perf_counter() - t)
            took.append(best)
    assert max(took[1:]) <= 3.0 * took[0], took
