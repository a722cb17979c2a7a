"""The density pass over states denser than its masks (k_density_mask) or its shared memory
(k_density_group: 64 members) have room for, which take several rounds: members and densities against a
brute-force evaluation, and a cost that grows with the candidates."""
import time

import numpy as np
import pytest

from test_gpu_density_filter import brute

pytestmark = pytest.mark.gpu


def lattice(dims, step):
    g = np.stack(np.meshgrid(*[np.arange(d) for d in dims], indexing="ij"), -1).reshape(-1, 3)
    return g * step


# (spacing of the particles, of the scene, cells in spacings, kernel in spacings)
STATES = {"two_rounds": (0.016, 0.02, 2.0, 2.0), "three_rounds": (0.0135, 0.02, 2.0, 2.0),
          "wide_kernel": (0.02, 0.02, 2.5, 2.5), "past_the_cap": (0.0092, 0.02, 2.0, 2.0)}


@pytest.mark.parametrize("name", list(STATES))
# sixteen lanes a particle, eight (up to 19,456), a row's records together (77,824), or one after another
@pytest.mark.parametrize("n", [1716, 9729, 19456, 20001, 77825])
def test_dense_members_and_density(gpu, name, n):
    import bubbles_gb300 as bb
    from bubbles_gb300 import scenes
    step, s, cells, kernel = STATES[name]
    r = np.random.default_rng(n)
    few = lattice((13, 12, 11), step)
    few = few - few.mean(0) + r.uniform(-0.1, 0.1, few.shape) * step
    m = len(few)
    rest = lattice((90, 30, 30), s)[:n - m] + np.array([1.0, -0.3, -0.3])
    pos = np.concatenate([few, rest]).astype(np.float32)
    sc = scenes.base_scene("pcisph", s, (6.0, 0.8, 0.8))
    sc.update(grid_spacing_scale=cells, relative_kernel_radius=kernel)
    with bb.Solver(sc, pos=pos) as q:
        assert q.n == n
        q.update_grid_distribution()
        cell, counts, _ = q.dump_grid()
        dims, _ = q.grid()
        q.compute_density(0)
        got_n, got = q.neighbor_lists(400)
        rho = q.get(bb.FIELD_DENSITY).astype(np.float64)
        scalars = q.scalars()
    h, mass = float(np.float32(scalars["kernel_radius"])), float(np.float32(scalars["mass"]))
    w = 315.0 / (64.0 * np.pi * h ** 3) * mass
    c27 = counts.reshape(dims[2], dims[1], dims[0]).astype(np.int64)
    near = np.flatnonzero(np.abs(pos[:, 0]) < 0.5)   # the dense block: the rest is out of its reach
    assert len(near) == m
    want = brute(pos[near], cell[near].astype(np.int64), dims, h)
    crowded = 0
    for i in range(m):
        x, y, z = int(cell[i] % dims[0]), int(cell[i] // dims[0] % dims[1]), int(cell[i] // (dims[0] * dims[1]))
        if c27[max(z - 1, 0):z + 2, max(y - 1, 0):y + 2, max(x - 1, 0):x + 2].sum() > 1024:   # the work cap
            want[i] = np.zeros(0, np.int64)
            crowded += 1
        assert got_n[i] == len(want[i]), i
        assert set(got[i, :got_n[i]]) == set(want[i]), i
        d2 = ((pos[want[i]].astype(np.float64) - pos[i].astype(np.float64)) ** 2).sum(1)
        ref = w * (1.0 + ((1.0 - d2 / h ** 2).clip(0) ** 3).sum())
        # positive terms added one after another, each with its own few roundings; the two constants
        assert abs(rho[i] - ref) <= (len(d2) + 20) * 2.0 ** -24 * ref, i
    assert (crowded > 0) == (name == "past_the_cap")


@pytest.mark.parametrize("side,step,cells,kernel", [(60, 0.85, 2.0, 2.0), (60, 1.0, 2.5, 2.5), (21, 0.8, 2.0, 2.0),
                                                    (25, 1.0, 3.0, 3.0)])
def test_cost_grows_with_the_candidates(gpu, side, step, cells, kernel):
    """The work of a particle is its candidates' tests and its members' sums: a state with k times the
    members takes k times as long, here at most 1.5 k times for what the rounds repeat."""
    import bubbles_gb300 as bb
    from bubbles_gb300 import scenes
    took, members = [], []
    for a, c, k in ((1.0, 2.0, 2.0), (step, cells, kernel)):
        s = 0.01
        g = lattice((side,) * 3, s * a)
        pos = (g - g.mean(0) + np.random.default_rng(1).uniform(-0.05, 0.05, g.shape) * s).astype(np.float32)
        sc = scenes.base_scene("pcisph", s, (1.4, 0.8, 0.8))
        sc.update(grid_spacing_scale=c, relative_kernel_radius=k)
        with bb.Solver(sc, pos=pos) as q:
            q.update_grid_distribution()
            best = float("inf")
            for _ in range(8):
                q.synchronize()
                t = time.perf_counter()
                for _ in range(20):
                    q.compute_density(0)
                q.synchronize()
                best = min(best, time.perf_counter() - t)
            took.append(best)
            members.append(float(q.neighbor_lists(0)[0].mean()))
    assert took[1] <= 1.5 * took[0] * members[1] / members[0], (took, members)
