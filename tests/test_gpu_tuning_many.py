"""Launch tuning where every knob acts (more than 77,824 particles): gather batches 2, 4 and 8 of the three
corrector passes, one and two particles a thread, block sizes, tile orders and the batches' work lists
give the bits of the default."""
import numpy as np
import pytest

import bubbles_gb300 as bb
from bubbles_gb300 import scenes

pytestmark = pytest.mark.gpu

SINGLE = [dict(batch_np=2), dict(batch_np=8), dict(batch_pd=2), dict(batch_pd=8), dict(batch_pf=2), dict(batch_pf=8),
          dict(particles_per_thread=2), dict(particles_per_thread=2, batch_pd=2, batch_pf=8, block_size=64),
          dict(particles_per_thread=2, batch_pd=8, batch_pf=2, block_size=256, tile_order=1),
          dict(tile_order=1), dict(block_size=64), dict(block_size=256, batch_np=8)]
BATCH = [dict(batch_worklist=w, batch_pd=a, batch_pf=b, particles_per_thread=p, block_size=t)
         for w, a, b, p, t in ((0, 2, 8, 1, 64), (0, 8, 2, 2, 128), (0, 4, 4, 2, 256), (1, 2, 2, 1, 128),
                               (1, 8, 8, 2, 64), (1, 4, 4, 2, 256), (2, 2, 8, 1, 256), (2, 8, 2, 2, 64),
                               (2, 4, 4, 1, 128))]


def block(dims, step, seed):
    g = np.stack(np.meshgrid(*[np.arange(d) for d in dims], indexing="ij"), -1).reshape(-1, 3)
    r = np.random.default_rng(seed)
    return (g - g.mean(0)) * step + r.uniform(-0.05, 0.05, g.shape) * step, r.normal(0, 0.4, g.shape)


def substeps(s, n):
    out = []
    for _ in range(n):
        st = s.advance_time_step(2e-4, stats=True)
        out.append(np.array([st["iterations"], st["crowded"]]))
        out += [np.asarray(a) for a in s.download()]
        out.append(s.get(bb.FIELD_PRESSURE))
    return out


@pytest.mark.parametrize("start", ["zero", "previous", "learned"])
def test_single_scene(gpu, start):
    pos, vel = block((61, 37, 41), 0.0196, 1)
    assert len(pos) > 77824
    sc = scenes.base_scene("pcisph", 0.02, (1.6, 1.0, 1.0))
    sc.update(max_iterations=6, max_density_error_ratio=0.01, pressure_init=start)
    if start == "learned":
        sc["mlp"] = {"train_substeps": 1, "batch": 1024}
    want = None
    for tuning in [dict()] + SINGLE:
        with bb.Solver(sc, pos=pos.astype(np.float32), vel=vel.astype(np.float32)) as s:
            s.set_tuning(**tuning)
            got = substeps(s, 3)
        want = want or got
        for a, b in zip(got, want):
            assert a.tobytes() == b.tobytes(), tuning
    assert max(int(a[0]) for a in want[::4]) > 1


def test_batch(gpu):
    sc = scenes.base_scene("pcisph", 0.02, (1.0, 1.0, 1.0))
    sc.update(max_iterations=8, max_density_error_ratio=0.01)
    boxes, pos, vel = [], [], []
    for k, (dims, step) in enumerate((((40, 30, 31), 0.0196), ((33, 29, 37), 0.02), ((17, 19, 23), 0.0193),
                                      ((5, 3, 4), 0.02))):
        p, v = block(dims, step, k)
        half = np.asarray(dims) * 0.012 + 0.04
        boxes.append((tuple(-half), tuple(half)))
        pos.append(p.astype(np.float32))
        vel.append(v.astype(np.float32))
    assert sum(len(p) for p in pos) > 77824
    want = None
    for tuning in [dict()] + BATCH:
        s = bb.BatchSolver(sc, boxes, pos, vel)
        s.set_tuning(**tuning)
        got = []
        for _ in range(3):
            s.advance_time_step(2e-4)
            got += [np.asarray(a) for a in s.scene_stats()] + [np.asarray(a) for a in s.download()]
        s.close()
        want = want or got
        for a, b in zip(got, want):
            assert a.tobytes() == b.tobytes(), tuning
    its = np.concatenate(want[::4])
    assert its.max() > 1
