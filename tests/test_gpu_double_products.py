"""The two-float evaluation of the reference's double products (kernel weights of the surface
field) rounds as the double does, over the whole range of weights: a node beside one particle has
the field 0.5 - (m / rho) W(d) (SPH), whose W is formed in double and rounded to float
(kernel.cpp:123-132)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [1e-3, 0.037, 0.5, 60.0])
def test_sph_field_of_isolated_particles(gpu, radius):
    import bubbles_gb300 as bb
    from bubbles_gb300 import scenes
    r = np.random.default_rng(3)
    f = np.float32
    h = f(radius)
    # one particle per 4 x 4 x 4 cells of the kernel radius: at most one within reach of a node
    side = 4.0 * float(h)
    k = np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = ((k + 0.5) * side - 16.0 * float(h) + r.uniform(-0.2, 0.2, k.shape) * side).astype(f)
    sc = scenes.base_scene("sph", float(h) / 2, (8 * side,) * 3)
    sc["colliders"] = []
    with bb.Solver(sc, pos=pos) as s:
        s.update_grid_distribution()
        s.compute_density(0)
        rho = s.get(bb.FIELD_DENSITY)
        mass = f(s.scalars()["mass"])
        nodes, org, sp, vals = s.particle_sdf("sph", float(h), float(h) / 3)
    ax = [f(org[q]) + f(sp[q]) * np.arange(nodes[q], dtype=f) for q in range(3)]
    field = vals.reshape(nodes[2], nodes[1], nodes[0])
    h2 = f(h * h)
    wc = 315.0 / (64.0 * 3.14159265358979323846 * float(f(h2 * h)))
    seen = 0
    for p, d in zip(pos, rho):
        i = [np.searchsorted(ax[q], p[q]) for q in range(3)]
        at = np.stack(np.meshgrid(*[np.arange(max(i[q] - 2, 0), min(i[q] + 2, nodes[q])) for q in range(3)],
                                  indexing="ij"), -1).reshape(-1, 3)
        e = [ax[q][at[:, q]] - p[q] for q in range(3)]
        dist = np.sqrt((e[0] * e[0] + e[1] * e[1]) + e[2] * e[2])
        d2 = dist * dist
        off = d2 - h2
        near = ~((np.abs(off) < f(1e-8)) | (off > 0))
        x = (f(1.0) - d2 / h2).astype(np.float64)
        w = np.where(near, (wc * x * x * x).astype(f), f(0))
        want = f(0.5) - (mass / d) * w
        got = field[at[:, 2], at[:, 1], at[:, 0]]
        inside = np.all([(ax[q][at[:, q]] <= f(4 * side)) for q in range(3)], axis=0) & near
        assert np.array_equal(got[inside], want[inside])
        seen += int(inside.sum())
    assert seen > 1000
