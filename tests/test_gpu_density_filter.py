"""The density pass's half-precision filter drops no member: neighbour sets and densities
against a brute-force float32 / float64 evaluation over the 27 cells the grid reports, where the
filter's cases meet: rows longer than a mask, lists longer than a row of masks, cells larger
than the kernel radius, particle counts off the record size, pairs at the kernel radius, and
particles outside the grid (clamped into it) or not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def brute(p, cell, dims, h):
    """Members of every particle other than itself: IsWithinStd in float32 over the 27 cells."""
    p = np.asarray(p, np.float32)
    iz = np.nextafter(np.float32(1e-8), np.float32(1)) if np.float64(np.float32(1e-8)) < 1e-8 else np.float32(1e-8)
    h2 = np.float32(h) * np.float32(h)
    c = np.stack([cell % dims[0], cell // dims[0] % dims[1], cell // (dims[0] * dims[1])], 1).astype(np.int64)
    out = []
    with np.errstate(invalid="ignore", over="ignore"):
        for i in range(len(p)):
            near = np.abs(c - c[i]).max(1) <= 1
            d = p[i] - p
            e2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
            r = np.sqrt(e2)
            out.append(np.flatnonzero(near & (r * r - h2 <= -iz) & (np.arange(len(p)) != i)))
    return out


def states():
    r = np.random.default_rng(7)
    box = np.array([0.6, 0.5, 0.6])
    def uniform(n, part):   # n particles in the low corner, `part` of the box each way
        return -box / 2 + 0.021 + r.random((n, 3)) * (box * part - 0.042)
    g = np.stack(np.meshgrid(*[np.arange(9)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.02
    shell = np.array([[0.04, 0, 0], [0.04 * (1 - 2e-7), 0, 0], [0, 0.0399999, 0], [0.0230940, 0.0230940, 0.0230940]])
    out = np.concatenate([uniform(300, 0.5), uniform(40, 0.3) + 3.0, uniform(20, 0.2) - 50.0])
    odd = uniform(333, 0.4)
    odd[5] = np.nan
    odd[6, 1] = np.inf
    return {"sparse": (uniform(97, 1.0), 2.0), "one": (uniform(1, 1.0), 2.0),
            "dense": (uniform(1203, 0.25), 2.0),        # rows past 32 slots, lists past 64 members
            "crowd": (uniform(1500, 0.12), 2.0),        # past the masks kept per particle
            "lattice": (-0.2 + g, 2.0),                 # pairs at exactly the kernel radius
            "radius": (np.concatenate([shell, [[0, 0, 0]], uniform(60, 0.5)]), 2.0),
            "wide_cells": (uniform(801, 0.5), 3.0), "outside": (out, 2.0), "not_finite": (odd, 2.0)}


@pytest.mark.parametrize("name", ["sparse", "one", "dense", "crowd", "lattice", "radius", "wide_cells", "outside",
                                  "not_finite"])
def test_members_and_density(gpu, name):
    import bubbles_gb300 as bb
    from bubbles_gb300 import scenes
    pos, scale = states()[name]
    sc = scenes.base_scene("pcisph", 0.02, (0.6, 0.5, 0.6))
    sc["grid_spacing_scale"] = scale
    pos = np.asarray(pos, np.float32)
    with bb.Solver(sc, pos=pos) as s:
        s.update_grid_distribution()
        cell, counts, _ = s.dump_grid()
        dims, _ = s.grid()
        s.compute_density(0)
        got_n, got = s.neighbor_lists(min(1024, 5 * len(pos)))   # at most 5 ids a particle of capacity are staged
        rho = s.get(bb.FIELD_DENSITY).astype(np.float64)
    h = np.float32(2.0) * np.float32(0.02)
    want = brute(pos, cell.astype(np.int64), dims, h)
    c27 = counts.reshape(dims[2], dims[1], dims[0]).astype(np.int64)
    w = 315.0 / (64.0 * np.pi * float(h) ** 3) * float(np.float32(sc["mass"]))
    for i in range(len(pos)):
        x, y, z = int(cell[i] % dims[0]), int(cell[i] // dims[0] % dims[1]), int(cell[i] // (dims[0] * dims[1]))
        total = c27[max(z - 1, 0):z + 2, max(y - 1, 0):y + 2, max(x - 1, 0):x + 2].sum()
        if total > 1024:   # the work cap: the particle keeps only itself
            want[i] = np.zeros(0, np.int64)
        assert got_n[i] == len(want[i]), i
        assert set(got[i, :got_n[i]]) == set(want[i]), i
        if not np.isfinite(pos[i]).all():
            continue
        d2 = ((pos[want[i]].astype(np.float64) - pos[i].astype(np.float64)) ** 2).sum(1)
        ref = w * (1.0 + ((1.0 - d2 / float(h) ** 2).clip(0) ** 3).sum())
        assert abs(rho[i] - ref) <= 1e-5 * ref, i
