"""Neighbour lists of few particles asked for with more room than they have staging for, and with
more than a particle can have members."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 10, 40, 171, 172])
@pytest.mark.parametrize("room", [0, 1, 7, 64, 1023, 1024, 1025, 5000])
def test_rows_of_any_width(gpu, n, room):
    import bubbles_gb300 as bb
    from bubbles_gb300 import scenes
    r = np.random.default_rng(n)
    pos = (r.random((n, 3)) * 0.08).astype(np.float32)
    with bb.Solver(scenes.base_scene("pcisph", 0.02, (0.4, 0.4, 0.4)), pos=pos) as s:
        s.update_grid_distribution()
        s.compute_density(0)
        h = np.float32(s.scalars()["kernel_radius"])
        count, ids = s.neighbor_lists(room)
    assert ids.shape == (n, room)
    d = np.sqrt(((pos[:, None] - pos[None]) ** 2).sum(2, dtype=np.float32))
    for i in range(n):
        want = np.flatnonzero((d[i] < h) & (np.arange(n) != i))   # no pair near the radius
        assert np.abs(np.delete(d[i], i) - h).min(initial=1.0) > 1e-7
        k = min(len(want), room)
        assert count[i] == len(want)
        assert set(ids[i, :k]) <= set(want) and len(set(ids[i, :k])) == k
        assert (ids[i, k:] == -1).all()
