"""The particle field where a node keeps more particles than fit its list, against a float64
evaluation; and meshes larger than the facade's first guess, against the two-call form of the C entry."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,size", [(1, 0.01), (59, 0.02), (61, 0.02), (3000, 0.05), (900, 0.3)])
def test_zhu_bridson_of_dense_particles(gpu, n, size):
    import bubbles_gb300 as bb
    from bubbles_gb300 import scenes
    r = np.random.default_rng(n)
    pos = ((r.random((n, 3)) - 0.5) * size).astype(np.float32)
    R, eps = float(np.float32(0.04)), 2.0 ** -24
    with bb.Solver(scenes.base_scene("sph", 0.02, (0.5, 0.5, 0.5)), pos=pos) as s:   # cells as wide as the radius
        s.update_grid_distribution()
        nodes, org, sp, v = s.particle_sdf("zhu", R, 0.0171)
    g = np.stack(np.meshgrid(*[np.arange(k) for k in nodes[::-1]], indexing="ij"), -1).reshape(-1, 3)[:, ::-1]
    p = org + g * sp
    x = pos.astype(np.float64)
    seen = 0
    for q, value in zip(p, v.astype(np.float64)):
        d = np.sqrt(((q - x) ** 2).sum(1))
        w = np.where(d < R, (1.0 - (d / R) ** 2).clip(0) ** 3, 0.0)
        near = int((d < 1.01 * R).sum())
        if w.sum() < 1e-3:
            assert near or value > 0.5   # nothing near: the grid's diagonal
            continue
        seen += 1
        want = np.sqrt(((q - (w[:, None] * x).sum(0) / w.sum()) ** 2).sum()) - 0.25 * R
        # sums of `near` rounded terms of size <= 0.25, and each weight's own rounding
        tol = (2 * near + 40) * eps + 10 * near * eps * 2 * R / w.sum()
        assert abs(value - want) <= tol
    assert seen > 0


@pytest.mark.parametrize("nodes", [(2, 2, 2), (3, 2, 5), (24, 25, 23)])
def test_meshes_of_noise(gpu, nodes):
    import bubbles_gb300 as bb
    from bubbles_gb300 import _native as N
    from bubbles_gb300 import scenes
    v = np.random.default_rng(2).normal(size=int(np.prod(nodes))).astype(np.float32)
    with bb.Solver(scenes.base_scene("sph", 0.02, (0.5, 0.5, 0.5)), pos=np.zeros((1, 3), np.float32)) as s:
        got = s.marching_cubes(nodes, (0, 0, 0), 0.1, v, 0.0)
        g = N.SdfGrid()
        for k in range(3):
            g.nodes[k], g.origin[k], g.spacing[k] = nodes[k], 0.0, 0.1
        a, b = ctypes.c_size_t(), ctypes.c_size_t()
        N.load().bbg_marching_cubes(s.h, ctypes.byref(g), v.ctypes.data, 0.0, 0, None, None, 0, None, 0,
                                    ctypes.byref(a), ctypes.byref(b))
        want = [np.empty((a.value, 3), np.float32), np.empty((a.value, 3), np.float32),
                np.empty((b.value, 3), np.int32)]
        N.call("bbg_marching_cubes", s.h, ctypes.byref(g), v.ctypes.data, 0.0, 0, want[0].ctypes.data,
               want[1].ctypes.data, a.value, want[2].ctypes.data, b.value, ctypes.byref(a), ctypes.byref(b))
    # every crossed edge has its vertex
    f = (v <= 0).reshape(nodes[::-1])
    assert a.value == sum(int((np.diff(f.astype(np.int8), axis=k) != 0).sum()) for k in range(3))
    for x, y in zip(got, want):
        assert x.shape == y.shape and x.dtype == y.dtype and x.tobytes() == y.tobytes()
