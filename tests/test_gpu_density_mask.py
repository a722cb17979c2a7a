"""The density pass's half-precision filter (k_density_mask, which more than 19,456 particles take) drops no
member: the states of test_gpu_density_filter.py, whose counts take the pass that has no filter, beside
enough other particles, in both forms of the filter (up to 77,824 particles and past them), with the
records written by the pass over set positions and by the grid update's gather."""
import numpy as np
import pytest

from test_gpu_density_filter import brute, states

pytestmark = pytest.mark.gpu

NAMES = ["sparse", "one", "dense", "crowd", "lattice", "radius", "wide_cells", "outside", "not_finite"]


def rest(n):
    g = np.stack(np.meshgrid(np.arange(120), np.arange(24), np.arange(28), indexing="ij"), -1).reshape(-1, 3)
    return g[:n] * 0.02 + np.array([0.5, -0.24, -0.28])


def expected(pos, m, cell, counts, dims, h):
    """Members of the first m particles, with the work cap: more than 1,024 candidates leave none."""
    c = np.stack([cell % dims[0], cell // dims[0] % dims[1], cell // (dims[0] * dims[1])], 1).astype(np.int64)
    c27 = counts.reshape(dims[2], dims[1], dims[0]).astype(np.int64)
    # a member is in one of the 27 cells: only the cells next to one of the m
    near = np.zeros(len(pos), bool)
    for lo in np.unique(c[:m], axis=0):
        near |= np.abs(c - lo).max(1) <= 1
    near[:m] = True
    idx = np.flatnonzero(near)   # ascending: the first m are themselves
    want = brute(pos[idx], cell[idx].astype(np.int64), dims, h)[:m]
    out = []
    for i in range(m):
        x, y, z = c[i]
        total = c27[max(z - 1, 0):z + 2, max(y - 1, 0):y + 2, max(x - 1, 0):x + 2].sum()
        out.append(np.zeros(0, np.int64) if total > 1024 else idx[want[i]])
    return out


@pytest.mark.parametrize("recorded", [False, True])
@pytest.mark.parametrize("n", [19457, 77824, 77825])
@pytest.mark.parametrize("name", NAMES)
def test_no_member_is_dropped(gpu, name, n, recorded):
    import bubbles_gb300 as bb
    from bubbles_gb300 import scenes
    few, scale = states()[name]
    m = len(few)
    pos = np.concatenate([few, rest(n - m)]).astype(np.float32)
    sc = scenes.base_scene("sph", 0.02, (6.2, 0.5, 0.6))
    sc["grid_spacing_scale"] = scale
    with bb.Solver(sc, pos=pos) as s:
        s.update_grid_distribution()
        cell, counts, _ = s.dump_grid()
        dims, _ = s.grid()
        if recorded:
            s.advance_time_step(1e-5)   # sorts the same positions again; its sets are the step-start ones
        else:
            s.compute_density(0)
        got_n, got = s.neighbor_lists(512)
        rho = s.get(bb.FIELD_DENSITY).astype(np.float64)
        scalars = s.scalars()
    h, mass = float(np.float32(scalars["kernel_radius"])), float(np.float32(scalars["mass"]))
    want = expected(pos, m, cell, counts, dims, np.float32(h))
    w = 315.0 / (64.0 * np.pi * h ** 3) * mass
    for i in range(m):
        assert got_n[i] == len(want[i]), i
        k = min(len(want[i]), 512)
        assert set(got[i, :k]) <= set(want[i]) and len(set(got[i, :k])) == k, i
        if not np.isfinite(pos[i]).all():
            continue
        d2 = ((pos[want[i]].astype(np.float64) - pos[i].astype(np.float64)) ** 2).sum(1)
        ref = w * (1.0 + ((1.0 - d2 / h ** 2).clip(0) ** 3).sum())
        # positive terms added one after another, each with its own few roundings, at least 1 in all; a
        # difference of coordinates rounds by half an ulp of itself
        assert abs(rho[i] - ref) <= (2 * len(d2) + 20) * 2.0 ** -24 * ref, i
