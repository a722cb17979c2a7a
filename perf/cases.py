"""Performance cases of bubbles_gb300: what a program that uses the solver has it do.

Each case is one pass through the public Python entry points on a fluid state made from a
seed: a dam break caught in motion (a jittered lattice block with a collapsing, locally
compressing velocity field, and a spray of droplets over the free part of the box).

    step      a PCISPH substep from a state on the device: upload, AdvanceTimeStep, download
    advance   SphSolver3::Advance over its CFL substeps, likewise
    batch     a PCISPH substep of many independent scenes advanced together
    learned   a substep with the learned warm start, state in pinned host memory
    train     one optimiser step of the warm-start network on a host batch
    mesh      the signed-distance field of a triangle mesh obstacle
    boundary  boundary classification of a particle frame
    surface   particles -> field -> marching-cubes mesh
    frame     a particle frame written as text and read back
"""
import math

import numpy as np
import torch

import bubbles_gb300 as bb
from bubbles_gb300 import scenes

PI = math.pi


def listed():
    return [
        # the smallest calls: a small ragged SPH scene (interactive preview, tests)
        {"name": "sph_1k", "kind": "advance", "dims": "11x9x13", "spacing": 0.02},
        # the repository's SPH dam break: 16,384 particles, Advance(1e-3) in 7 CFL substeps
        {"name": "sph_16k", "kind": "advance", "dims": "32x16x32", "spacing": 0.02},
        # its PCISPH dam break of 262,144 particles with a sphere, at its CFL substep
        {"name": "pcisph_262k", "kind": "step", "dims": "64x64x64", "spacing": 0.01, "dt_scale": 0.625,
         "spheres": 1, "cap": 20, "press": 0.5},
        # its 1M dam break at the long substep of the tolerance corrector (several iterations)
        {"name": "pcisph_1m", "kind": "step", "dims": "128x64x128", "spacing": 0.008, "dt_scale": 1.0,
         "spheres": 0, "cap": 64, "press": 5.0},
        # its largest scene: 4,194,304 particles, 8 spheres
        {"name": "pcisph_4m", "kind": "step", "dims": "256x64x256", "spacing": 0.005, "dt_scale": 0.625,
         "spheres": 8, "cap": 20, "press": 0.5},
        # its batch: 64 uneven scenes of 8k to 131k particles in one solver
        {"name": "batch_64", "kind": "batch", "scenes": 64, "nmin": 8192, "nmax": 131072, "spacing": 0.01,
         "cap": 64, "press": 5.0},
        # the learned warm start as a host program drives it (the benchmark's end-to-end step)
        {"name": "learned_1m", "kind": "learned", "dims": "128x64x128", "spacing": 0.008, "cap": 64, "press": 5.0},
        # online training of the warm start: the default batch of 16,384 pairs
        {"name": "train_16k", "kind": "train", "batch": 16384},
        # an obstacle's field at scene setup: a torus of 1,152 triangles, about 0.2M nodes
        {"name": "mesh_torus", "kind": "mesh", "nu": 32, "nv": 18, "dx": 0.011},
        # post-processing of a frame of 262,144 particles: Xiaowei's boundary test
        {"name": "xiaowei_262k", "kind": "boundary", "dims": "64x64x64", "spacing": 0.01, "test": "xiaowei"},
        # the surface of the same frame (Zhu-Bridson field, marching cubes)
        {"name": "surface_262k", "kind": "surface", "dims": "64x64x64", "spacing": 0.01},
        # the same frame to text and back
        {"name": "frame_262k", "kind": "frame", "dims": "64x64x64", "spacing": 0.01},
    ]


def _block(rng, lo, hi):
    """Ragged block dimensions of about n particles, n log-uniform in [lo, hi]."""
    while True:
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        a = [rng.uniform(0.4, 1.0) for _ in range(3)]
        k = (n / (a[0] * a[1] * a[2])) ** (1.0 / 3.0)
        d = [max(4, int(round(x * k))) for x in a]
        if d[0] * d[1] * d[2] <= hi:
            return "%dx%dx%d" % tuple(d)


def _dims(case):
    return [int(x) for x in case["dims"].split("x")]


def draw(rng):
    kind = rng.choice(["advance", "step", "step", "step", "batch", "learned", "train", "mesh", "boundary", "surface",
                       "frame"])
    h0 = rng.choice([0.005, 0.008, 0.01, 0.02])
    if kind == "advance":
        return {"kind": kind, "dims": _block(rng, 1000, 16384), "spacing": 0.02}
    if kind == "step":
        long = rng.random() < 0.5
        return {"kind": kind, "dims": _block(rng, 2000, 1048576 if long else 4194304), "spacing": h0,
                "dt_scale": 1.0 if long else 0.625, "spheres": rng.choice([0, 1, 8]), "cap": 64 if long else 20,
                "press": 5.0 if long else 0.5}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 64), "nmin": 1500, "nmax": rng.choice([8192, 30000, 65536]),
                "spacing": 0.01, "cap": 64, "press": 5.0}
    if kind == "learned":
        return {"kind": kind, "dims": _block(rng, 4000, 1048576), "spacing": h0, "cap": 64, "press": 5.0}
    if kind == "train":
        return {"kind": kind, "batch": int(math.exp(rng.uniform(math.log(500), math.log(16384))))}
    if kind == "mesh":
        return {"kind": kind, "nu": rng.randint(6, 32), "nv": rng.randint(5, 18), "dx": rng.uniform(0.0115, 0.04)}
    dims = _block(rng, 3000, 262144)
    if kind == "boundary":
        t = rng.choice(["xiaowei", "dilts", "lnm", "lnm_single", "lnm_extended", "lnm_xiaowei"])
        return {"kind": kind, "dims": _block(rng, 3000, 95000) if t == "dilts" else dims, "spacing": h0, "test": t}
    return {"kind": kind, "dims": dims, "spacing": h0}


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    g = torch.Generator(device=_dev())
    g.manual_seed(int(seed) % (1 << 31) + 17)
    return g


def _box(case):
    """Container of the block: twice its x and 1.5 times its y extent, as a dam break has."""
    d, s = _dims(case), case["spacing"]
    return np.array([2.0 * (1.02 * d[0] + 2) * s, 1.5 * (1.02 * d[1] + 2) * s, (1.02 * d[2] + 4) * s])


def _scene(case):
    """The scene dict of a single-scene case (spheres on the floor of the free half)."""
    d, s = _dims(case), case["spacing"]
    kind = "sph" if case["kind"] == "advance" else "pcisph"
    box = _box(case)
    sc = scenes.base_scene(kind, s, tuple(box))
    sc.update(max_iterations=case.get("cap", 20), max_density_error_ratio=0.01)
    n = case.get("spheres", 0)
    for k in range(n):
        r = min(0.08 * box[0], 0.3 * box[1], 0.4 * box[2] / max(1, n // 2))
        x = (0.18 + 0.22 * (k % 2)) * box[0]
        z = (-0.5 + (k // 2 + 0.5) / max(1, (n + 1) // 2)) * box[2]
        sc["colliders"].append({"type": "sphere", "center": (float(x), float(-0.5 * box[1] + r), float(z)),
                                "radius": float(r)})
    return sc


def _state(dims, s, lo, box, press, g, bcc=False):
    """(positions, velocities) float32 of a block at `lo` inside its container of size `box`:
    the block, near its rest density, in a collapsing flow whose local compression is `press`
    percent a substep at the speed limit (which sets the corrector's iterations: one at 0.5,
    about five at 5), 1 % of the particles as spray over the free part of the box.  `bcc`: the volume
    emitter's lattice (which the Dilts test is made for) instead of the cubic one."""
    dev = _dev()
    nx, ny, nz = dims
    ax = [torch.arange(m, device=dev, dtype=torch.float64) for m in (nz, ny, nx)]
    z, y, x = torch.meshgrid(*ax, indexing="ij")
    p = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)
    n = len(p)
    u = (p + 0.5) / torch.tensor([nx, ny, nz], device=dev, dtype=torch.float64)   # 0..1 in the block
    jit = torch.rand((n, 3), generator=g, device=dev, dtype=torch.float64) * 2 - 1
    low = torch.tensor(lo, device=dev, dtype=torch.float64)
    if bcc:   # the volume emitter's lattice: layers half a spacing apart, every other one shifted
        odd = 0.5 * (p[:, 2] % 2)
        p = torch.stack([p[:, 0] + odd, p[:, 1] + odd, 0.5 * p[:, 2]], 1)
    pos = low + s * (1.0 + 1.02 * p + 0.05 * jit)
    # collapse: the top sinks, the front runs out; waves of compression along the three axes
    dt = 0.4 * (2 * s) / 100.0 * 5.0
    v = torch.stack([1.5 * u[:, 0] * (0.3 + u[:, 1]), -1.0 * u[:, 1], torch.zeros_like(u[:, 0])], 1)
    k = 2 * PI / 12.0                          # wave length: 12 spacings
    amp = 0.01 * press / (3 * dt * k / s)      # div v dt = press % at the crests
    ph = 2 * PI * torch.rand(3, generator=g, device=dev, dtype=torch.float64)
    v = v + amp * torch.sin(k * p + ph)
    v = v + 0.02 * torch.randn((n, 3), generator=g, device=dev, dtype=torch.float64)
    # spray: every 100th particle somewhere in the free part, falling
    m = torch.arange(37 % max(1, n), n, 100, device=dev)
    r = torch.rand((len(m), 3), generator=g, device=dev, dtype=torch.float64)
    b = torch.tensor(box, device=dev, dtype=torch.float64)
    free = torch.tensor([(1.02 * nx + 4) * s, 0.0, 0.0], device=dev, dtype=torch.float64)
    pos[m] = low + 1.1 * s + free + r * (b - 2.2 * s - free).clamp_min(0.5 * s)
    v[m] = v[m] + torch.tensor([0.5, -1.0, 0.0], device=dev, dtype=torch.float64)
    return pos.float().contiguous(), v.float().contiguous()


def _single(case, seed):
    box = _box(case)
    g = _gen(seed)
    pos, vel = _state(_dims(case), case["spacing"], list(-box / 2), list(box), case.get("press", 0.5), g,
                      case.get("test") == "dilts")
    return pos, vel, g


def _dt(case):
    return 1e-3 if case["kind"] == "advance" else 0.4 * (2 * case["spacing"]) / 100.0 * 5.0 * case.get("dt_scale", 1.0)


def _theta(seed):
    """Warm-start weights as training leaves them: mostly the previous pressure and the local
    compression, through two of the hidden units, among small ones."""
    r = np.random.default_rng(seed)
    w1, b1 = 0.1 * r.standard_normal((4, 64)), 0.02 * r.standard_normal(64)
    w2, b2 = 0.1 * r.standard_normal((64, 64)), 0.02 * r.standard_normal(64)
    w3, b3 = 0.02 * r.standard_normal(64), np.zeros(1)
    w1[:, 0] = (0.4, 0.3, 0.0, 0.8)
    b1[0] = 0.0
    w2[:, 0] = 0.0
    w2[0, 0] = 1.0
    w3[0] = 1.0
    return np.concatenate([w1.ravel(), b1, w2.ravel(), b2, w3, b3]).astype(np.float32)


def _carried(case, n, g, p_unit):
    """The carried pressure and divergence of a learned run: pressure from the floor up to the
    surface, at most 2 p_unit, and a divergence sum of a few percent of a substep."""
    dev, d = _dev(), _dims(case)
    y = (torch.arange(n, device=dev) // d[0] % d[1]).double() / d[1]
    p = p_unit * (2.0 * (1.0 - y) + 0.05 * torch.randn(n, generator=g, device=dev, dtype=torch.float64)).clamp_min(0.0)
    dv = 0.01 * torch.randn(n, generator=g, device=dev, dtype=torch.float64)
    return p.float(), dv.float()


def _mesh(case, seed):
    """A tilted torus (radii 0.3 and 0.1) of nu x nv quads, its tube dented by up to 10 % from the
    seed everywhere but at the vertices that set its bounds."""
    nu, nv = case["nu"], case["nv"]
    u, w = np.meshgrid(2 * np.pi * np.arange(nu) / nu, 2 * np.pi * np.arange(nv) / nv, indexing="ij")
    v = np.stack([(0.3 + 0.1 * np.cos(w)) * np.cos(u), (0.3 + 0.1 * np.cos(w)) * np.sin(u), 0.1 * np.sin(w)],
                 axis=-1).reshape(-1, 3)
    a, b, c = 0.5, 0.9, 0.3
    rx = np.array([[1, 0, 0], [0, np.cos(a), -np.sin(a)], [0, np.sin(a), np.cos(a)]])
    ry = np.array([[np.cos(b), 0, np.sin(b)], [0, 1, 0], [-np.sin(b), 0, np.cos(b)]])
    rz = np.array([[np.cos(c), -np.sin(c), 0], [np.sin(c), np.cos(c), 0], [0, 0, 1]])
    rot = (rx @ ry @ rz).T
    mid = np.stack([0.3 * np.cos(u), 0.3 * np.sin(u), 0 * u], -1).reshape(-1, 3)
    t = v @ rot
    fix = np.unique(np.concatenate([t.argmin(0), t.argmax(0)]))
    dent = np.random.default_rng(seed).uniform(0.9, 1.0, (len(v), 1))
    dent[fix] = 1.0
    v = ((mid + dent * (v - mid)) @ rot).astype(np.float32)
    i, j = np.meshgrid(np.arange(nu), np.arange(nv), indexing="ij")
    p, q = i * nv + j, ((i + 1) % nu) * nv + j
    r, t = ((i + 1) % nu) * nv + (j + 1) % nv, i * nv + (j + 1) % nv
    tri = np.stack([np.stack([p, q, r], -1), np.stack([p, r, t], -1)], 2).reshape(-1, 3).astype(np.int32)
    return v, tri


def _pairs(case, seed):
    r = np.random.default_rng(seed)
    n = case["batch"]
    f = np.stack([2 * r.standard_normal(n), 3 * r.standard_normal(n), r.uniform(0.5, 1.1, n),
                  np.maximum(2 + 1.5 * r.standard_normal(n), 0)], 1).astype(np.float32)
    t = np.maximum(0.5 * f[:, 0] + 0.3 * f[:, 1] + 0.8 * f[:, 3] + 0.2 * r.standard_normal(n), 0).astype(np.float32)
    return f, t


def _batch(case, seed):
    """(boxes, dims) of the batch's scenes, fixed by the case's sizes, not by the seed."""
    return _scene_dims(case["scenes"], case["nmin"], case["nmax"], case["spacing"])


def _scene_dims(count, nmin, nmax, s):
    r = np.random.default_rng(count * 7919 + nmax)
    boxes, dims = [], []
    for _ in range(count):
        n = math.exp(r.uniform(math.log(nmin), math.log(nmax)))
        a = r.uniform(0.3, 1.0, 3)
        k = (n / float(np.prod(a))) ** (1.0 / 3.0)
        d = [max(3, int(round(x))) for x in a * k]
        ext = 1.02 * np.array([2.0 * d[0] * s, 1.5 * d[1] * s, d[2] * s]) + 4.0 * s
        boxes.append((tuple(-ext / 2), tuple(ext / 2)))
        dims.append(d)
    return boxes, dims


def _packed(boxes, s):
    """Where a batch places its containers: stacked along z, each from a cell boundary, two
    empty cells apart (the offsets BatchSolver.layout() reports)."""
    cell, z, off = 2.0 * s, 0.0, []
    for lo, hi in boxes:
        off.append([-lo[0], -lo[1], z - lo[2]])
        z = math.ceil((z + hi[2] - lo[2]) / cell) * cell + 2.0 * cell
    return off


def _batch_state(case, seed):
    boxes, dims = _batch(case, seed)
    off = _packed(boxes, case["spacing"])
    g = _gen(seed)
    pos, vel = [], []
    for (lo, hi), d, o in zip(boxes, dims, off):
        p, v = _state(d, case["spacing"], [lo[k] + o[k] for k in range(3)], [hi[k] - lo[k] for k in range(3)],
                      case["press"], g)
        pos.append(p)
        vel.append(v)
    return pos, vel


def _pinned(t):
    return torch.empty(t.shape, dtype=torch.float32, pin_memory=True).copy_(t).numpy()


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "kind": kind}
    if kind == "train":
        s = bb.PciSphSolver3(dict(scenes.base_scene("pcisph", 0.01, (1.0, 1.0, 1.0)), pressure_init="learned"),
                             capacity=max(1024, case["batch"]))
        s.mlp_set_params(_theta(seed))
        st["pairs"] = _pairs(case, seed)
    elif kind == "mesh":
        sc = scenes.base_scene("pcisph", 0.02, (2.0, 2.0, 2.0))
        s = bb.PciSphSolver3(sc, capacity=16)
        st["mesh"] = _mesh(case, seed)
    elif kind == "batch":
        pos, vel = _batch_state(case, seed)
        boxes, _ = _batch(case, seed)
        sc = scenes.base_scene("pcisph", case["spacing"], (1.0, 1.0, 1.0))
        sc.update(max_iterations=case["cap"], max_density_error_ratio=0.01)
        s = bb.BatchSolver(sc, boxes, [np.zeros((len(p), 3), np.float32) for p in pos], setup=True)
        st["pos"], st["vel"] = torch.cat(pos), torch.cat(vel)
    else:
        pos, vel, g = _single(case, seed)
        sc = _scene(case)
        n = len(pos)
        if kind == "learned":
            sc.update(pressure_init="learned")
        s = (bb.SphSolver3 if kind == "advance" else bb.PciSphSolver3)(sc, capacity=n)
        torch.cuda.synchronize()
        s.upload_device(pos, vel)
        s.setup()
        if kind == "learned":
            s.mlp_set_params(_theta(seed))
            s.mlp_set_trained(200)
            press, div = _carried(case, n, g, _delta(sc, _dt(case)) * 10.0)
            st["in"] = [_pinned(a) for a in (pos, vel, press, div)]
            st["out"] = [_pinned(torch.zeros_like(a)) for a in (pos, vel, press, div)]
        if kind == "frame":
            st["reader"] = bb.PciSphSolver3(sc, capacity=n)
            st["text"] = bytearray(96 * n + 512)
        if kind == "surface":
            st["mesh"] = [np.zeros((n, 3), np.float32), np.zeros((n, 3), np.float32), np.zeros((2 * n, 3), np.int32)]
        st["pos"], st["vel"] = pos, vel
    st["solver"] = s
    if "pos" in st:
        st["pos_out"], st["vel_out"] = torch.empty_like(st["pos"]), torch.empty_like(st["vel"])
    s.synchronize()
    torch.cuda.synchronize()
    return st


def run(st):
    s, case, kind = st["solver"], st["case"], st["kind"]
    if kind in ("step", "batch"):
        s.upload_device(st["pos"], st["vel"])
        s.advance_time_step(_dt(case))
        s.download_device(st["pos_out"], st["vel_out"])
        return {"pos": st["pos_out"], "vel": st["vel_out"]}
    if kind == "advance":
        s.upload_device(st["pos"], st["vel"])
        got = s.advance(_dt(case))
        s.download_device(st["pos_out"], st["vel_out"])
        return {"pos": st["pos_out"], "vel": st["vel_out"], "substeps": got["substeps"]}
    if kind == "learned":
        s.step_host(_dt(case), *st["in"], *st["out"])
        return dict(zip(("pos", "vel", "pressure", "divergence"), st["out"]))
    if kind == "train":
        s.mlp_train_batch(*st["pairs"])
        return {"theta": s.mlp_params()}
    if kind == "mesh":
        nodes, org, sp, vals, _, stuck = s.mesh_sdf(*st["mesh"], dx=case["dx"], margin=0.1)
        return {"nodes": nodes, "origin": org, "spacing": sp, "values": vals, "stuck": stuck}
    s.upload_device(st["pos"], st["vel"])
    h = case["spacing"]
    if kind == "boundary":
        s.update_grid_distribution()
        t = case["test"]
        if t == "xiaowei":
            s.compute_density(0)
            return {"boundary": s.boundary_test("xiaowei", h)}
        if t == "dilts":
            return {"boundary": s.boundary_test("dilts")}
        if t == "lnm_xiaowei":
            s.compute_density(0)
            levels, queued, accepted = s.lnm_boundary_geometric(h, "xiaowei")
            return {"levels": levels, "queued": queued, "accepted": accepted}
        return {"levels": {"lnm": s.lnm_boundary, "lnm_single": s.lnm_boundary_single,
                           "lnm_extended": s.lnm_boundary_extended}[t](h)}
    if kind == "surface":
        s.update_grid_distribution()
        nodes, org, sp, vals = s.particle_sdf("zhu", 2 * h, h)
        mesh = s.marching_cubes(nodes, org, sp, vals, 0.0)
        for buf, a in zip(st["mesh"], mesh):   # a renderer's buffers of fixed size
            buf[:len(a)] = a
            buf[len(a):] = 0
        return {"nodes": nodes, "values": vals, **dict(zip(("points", "normals", "triangles"), st["mesh"]))}
    flags = bb.FRAME_POSITION | bb.FRAME_VELOCITY
    size = s.frame_text(flags, out=st["text"])
    r = st["reader"]
    r.frame_load(bytes(memoryview(st["text"])[:size]), flags)
    r.download_device(st["pos_out"], st["vel_out"])
    return {"text": np.frombuffer(st["text"], np.uint8), "pos": st["pos_out"], "vel": st["vel_out"]}


def work(case):
    """Bytes: each particle's (node's, pair's) inputs and results once.  Operations: the sums
    over the 28 neighbours of each pass a substep cannot do without (corrector iterations:
    one at the CFL substep, five at the long one)."""
    kind = case["kind"]
    if kind == "train":
        return {"bytes": 20 * case["batch"] + 4 * 4545, "flops": 6 * case["batch"] * (4 * 64 + 64 * 64 + 64)}
    if kind == "mesh":
        nodes = 1.3 * 1.3 * 0.9 / case["dx"] ** 3 * 0.5
        return {"bytes": 4 * nodes + 36 * 2 * case["nu"] * case["nv"], "flops": 200 * nodes}
    if kind == "batch":
        _, dims = _batch(case, 0)
        n = sum(a * b * c for a, b, c in dims)
    else:
        n = math.prod(_dims(case))
    if kind in ("boundary", "frame", "surface"):
        return {"bytes": {"boundary": 16, "frame": 24 + 75 + 24, "surface": 12 + 4 * 0.4}[kind] * n,
                "flops": {"boundary": 216 * 12, "frame": 200, "surface": 300}[kind] * n}
    if kind == "advance":
        return {"bytes": 48 * n, "flops": 7 * 28 * 50 * n}
    it = 5 if case["press"] > 1.0 else 1
    return {"bytes": (64 if kind == "learned" else 48) * n, "flops": (28 * (40 + 30 * it) + (8700 if kind == "learned" else 0)) * n}


# ----------------------------------------------------------------------------
# the same in 64 bits
# ----------------------------------------------------------------------------
def _f(x):
    return float(np.float32(x))


def _delta(sc, dt):
    """ComputeDelta: -1 / (beta sum terms) over the BCC lattice of the kernel's support."""
    s, h = _f(sc["spacing"]), 2.0 * _f(sc["spacing"])
    a, half = 1.5 * h, 0.5 * s
    g1, g2 = np.zeros(3), 0.0
    for k in range(int(math.floor(2 * a / half + 1e-6)) + 1):
        off = half if k % 2 else 0.0
        m = int(math.floor((2 * a - off) / s + 1e-6)) + 1
        for j in range(m):
            for i in range(m):
                p = np.array([i * s + off - a, j * s + off - a, k * half - a])
                d = math.sqrt(float(p @ p))
                if 0.0 < d < h * (1 - 1e-7):
                    g = p / d * (45.0 / (PI * h ** 4) * (1 - d / h) ** 2)
                    g1 += g
                    g2 += float(g @ g)
    return 1.0 / (2.0 * (_f(sc["mass"]) / 1000.0) ** 2 * _f(dt) ** 2 * (float(g1 @ g1) + g2))


def _near(x, q, h):
    """All (query, particle) pairs closer than h, int64, by cells of size h."""
    lo = torch.minimum(x.min(0).values, q.min(0).values) - h
    dim = ((torch.maximum(x.max(0).values, q.max(0).values) - lo) / h).floor().long() + 2
    cell = lambda p: ((p - lo) / h).floor().long()  # noqa: E731
    key = lambda c: c[:, 0] + dim[0] * (c[:, 1] + dim[1] * c[:, 2])  # noqa: E731
    order = torch.argsort(key(cell(x)))
    keys, xs, cq = key(cell(x))[order], x[order], cell(q)
    ii, jj = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            c = cq + torch.tensor([-1, dy, dz], device=x.device)
            first, last = torch.searchsorted(keys, key(c)), torch.searchsorted(keys, key(c) + 3)
            for r in range(int((last - first).max()) if len(q) else 0):
                i = torch.nonzero(first + r < last).flatten()
                j = first[i] + r
                d2 = ((q[i] - xs[j]) ** 2).sum(1)
                hit = d2 < h * h
                ii.append(i[hit])
                jj.append(order[j[hit]])
    return torch.cat(ii), torch.cat(jj)


def _collide(x, v, rest, sc):
    """ResolveCollision: the nearest collider's surface; inside it or closer than the radius,
    the position moves out to the radius and the normal velocity is reflected by `rest`."""
    r = _f(sc["spacing"])
    best, bd = None, None
    for c in sc["cols"]:
        if "half" in c:   # the container, from inside
            p, hf = x - c["center"], c["half"]
            gap = hf - p.abs()
            k = gap.argmin(1, keepdim=True)
            ins = (gap >= 0).all(1)
            out = torch.zeros_like(p).scatter_(1, k, 1.0) * torch.where(p < 0, -1.0, 1.0)
            at_in = p + out * gap.gather(1, k)
            at = torch.where(ins[:, None], at_in, torch.maximum(torch.minimum(p, hf), -hf))
            ko = (p - at).abs().argmax(1, keepdim=True)
            nrm = torch.where(ins[:, None], out, torch.zeros_like(p).scatter_(1, ko, 1.0) * torch.where(p < 0, -1.0, 1.0))
            d = (p - at).norm(dim=1)
            got = (d, at + c["center"], -nrm, ~ins)
        else:
            p = x - c["center"]
            l = p.norm(dim=1)
            nrm = p / l[:, None]
            got = ((l - c["radius"]).abs(), c["center"] + nrm * c["radius"], nrm, l < c["radius"])
        if best is None:
            best, bd = got, got[0]
        else:
            w = got[0] < bd
            bd = torch.where(w, got[0], bd)
            best = tuple(torch.where(w if a.dim() == 1 else w[:, None], b, a) for a, b in zip(best, got))
    d, at, nrm, inside = best
    hit = inside | (d < r)
    vn = (v * nrm).sum(1, keepdim=True)
    vr = torch.where(vn < 0, v - (1 + rest) * vn * nrm, v)
    return torch.where(hit[:, None], at + r * nrm, x), torch.where(hit[:, None], vr, v)


def _colliders(sc, dev):
    t = lambda a: torch.tensor([_f(z) for z in a], device=dev, dtype=torch.float64)  # noqa: E731
    sc["cols"] = [{"center": t(c["center"]), "half": t(c["size"]) / 2} if c["type"] == "box" else
                  {"center": t(c["center"]), "radius": _f(c["radius"])} for c in sc["colliders"]]


def _substep(x, v, sc, dt, start=None, scene=None):
    """One substep in 64 bits: SPH (density, pressure from the equation of state, forces) or
    PCISPH (start(rho, count) -> start pressure or None; per-scene convergence)."""
    n, dev = len(x), x.device
    s = _f(sc["spacing"])
    h, m, rho0, dt = 2.0 * s, _f(sc["mass"]), 1000.0, _f(dt)
    i, j = _near(x, x, h)
    keep = i != j
    i, j = i[keep], j[keep]
    add = lambda w, dims: torch.zeros(dims, device=dev, dtype=torch.float64).index_add_(0, i, w)  # noqa: E731
    c_std = 315.0 / (64.0 * PI * h ** 3) * m
    e = x[j] - x[i]
    d = e.norm(dim=1)
    u = 1 - d / h
    rho = c_std * (1 + add((1 - (d / h) ** 2) ** 3, n))
    grav = torch.tensor([0.0, _f(-9.81), 0.0], device=dev, dtype=torch.float64)
    f = m * grav - _f(1e-4) * v + add((v[j] - v[i]) * (_f(0.04) * m * m * 90.0 / (PI * h ** 5) * u / rho[j])[:, None], (n, 3))
    g = e * (m * m * 45.0 / (PI * h ** 4) * u * u / d.clamp_min(1e-300))[:, None]
    div = add((u * u / d.clamp_min(1e-300) / rho[j]) * ((v[j] - v[i]) * e).sum(1), n)

    def pforce(p, r):
        a = p / (r * r)
        return -add(g * (a[i] + a[j])[:, None], (n, 3))

    def integrate(ft):
        w = v + ft / m * dt
        y, w = _collide(x + w * dt, w, _f(0.6), sc)
        return y, w

    if sc["solver"] == "sph":
        p = (rho0 * 100.0 ** 2 / 7.0 * ((rho / rho0) ** 7 - 1)).clamp_min(0.0)
        f = f + pforce(p, rho)
        y, w = integrate(f)
        return y, w, f, None, None
    delta = _delta(sc, dt)
    p = start(rho, torch.bincount(i, minlength=n)) if start else torch.zeros_like(rho)
    fp = pforce(p, rho) if start else torch.zeros_like(x)
    sid = torch.zeros(n, device=dev, dtype=torch.long) if scene is None else scene
    live = torch.ones(n, device=dev, dtype=torch.bool)
    y, w = x.clone(), v.clone()
    pairs = (i, j)
    for k in range(int(sc["max_iterations"])):
        xs = _collide(x + (v + (f + fp) * (dt / m)) * dt, v, 0.0, sc)[0]
        q = (1 - ((xs[pairs[1]] - xs[pairs[0]]) ** 2).sum(1) / (h * h)).clamp_min(0.0) ** 3
        rs = c_std * (1 + add(q, n))
        err = (rs - rho0).clamp_min(0.0)
        p = torch.where(live, p + delta * err, p)
        fn = pforce(p, rs)
        fp = torch.where(live[:, None], fn, fp)
        worst = torch.zeros(int(sid.max()) + 1, device=dev, dtype=torch.float64).scatter_reduce_(0, sid, err, "amax")
        done = live & ((worst < 0.01 * rho0)[sid] | (k == int(sc["max_iterations"]) - 1))
        yn, wn = integrate(f + fp)
        y, w = torch.where(done[:, None], yn, y), torch.where(done[:, None], wn, w)
        live = live & ~done
        if not bool(live.any()):
            break
    return y, w, f + fp, p, div


def _exact_step(case, seed):
    dev, dt, kind = _dev(), _dt(case), case["kind"]
    if kind == "batch":
        boxes, dims = _batch(case, seed)
        off = _packed(boxes, case["spacing"])
        pos, vel = _batch_state(case, seed)
        ys, ws = [], []
        for (lo, hi), o, p, v in zip(boxes, off, pos, vel):
            sc = scenes_like(case, [hi[k] - lo[k] for k in range(3)], [o[k] + 0.5 * (lo[k] + hi[k]) for k in range(3)])
            _colliders(sc, dev)
            y, w, _, _, _ = _substep(p.double(), v.double(), sc, dt)
            ys.append(y)
            ws.append(w)
        return {"pos": torch.cat(ys), "vel": torch.cat(ws)}
    pos, vel, g = _single(case, seed)
    sc = _scene(case)
    _colliders(sc, dev)
    x, v = pos.double(), vel.double()
    if kind == "advance":
        left, steps, fmax = _f(dt), 0, 0.0
        while left > 1e-4:
            h = 2.0 * _f(case["spacing"])
            lim = 0.4 * h / 100.0
            if fmax > 1e-8:
                lim = min(lim, 0.25 * math.sqrt(h * _f(sc["mass"]) / fmax))
            step = left / max(1, math.ceil(np.float32(left) / np.float32(lim)))
            x, v, f, _, _ = _substep(x, v, sc, step)
            fmax = float(f.norm(dim=1).max())
            left -= step
            steps += 1
        return {"pos": x, "vel": v, "substeps": None}
    start = None
    if kind == "learned":
        unit = _delta(sc, dt) * 10.0
        press, dprev = (a.double() for a in _carried(case, len(x), g, _delta(sc, dt) * 10.0))
        th = torch.tensor(_theta(seed), device=dev, dtype=torch.float64)
        w1, b1, w2, b2, w3, b3 = th.split([256, 64, 4096, 64, 64, 1])
        gelu = lambda z: torch.nn.functional.gelu(z, approximate="tanh")  # noqa: E731

        def start(rho, count):
            fe = torch.stack([100 * (rho / 1000.0 - 1),
                              -100 * _f(dt) * _f(sc["mass"]) * 45.0 / (PI * (2 * _f(sc["spacing"])) ** 4) * dprev,
                              count.double() / 32, press / unit], 1)
            z = gelu(gelu(fe @ w1.view(4, 64) + b1) @ w2.view(64, 64) + b2) @ w3 + b3
            return 0.9 * unit * z.clamp_min(0.0)

    y, w, _, p, div = _substep(x, v, sc, dt, start)
    if kind == "learned":
        return {"pos": y, "vel": w, "pressure": p, "divergence": div}
    return {"pos": y, "vel": w}


def scenes_like(case, size, center):
    """A PCISPH scene of one container of the batch, in the packed frame."""
    sc = scenes.base_scene("pcisph", case["spacing"], tuple(size))
    sc["colliders"] = [{"type": "box", "size": tuple(size), "center": tuple(center), "reverse": True}]
    sc.update(max_iterations=case["cap"])
    return sc


def _exact_train(case, seed):
    """One Adam step (learning rate 1e-3) on the mean squared error from zero moments."""
    f, t = (torch.tensor(a, dtype=torch.float64) for a in _pairs(case, seed))
    th = torch.tensor(_theta(seed), dtype=torch.float64, requires_grad=True)
    w1, b1, w2, b2, w3, b3 = th.split([256, 64, 4096, 64, 64, 1])
    gelu = lambda z: torch.nn.functional.gelu(z, approximate="tanh")  # noqa: E731
    y = gelu(gelu(f @ w1.view(4, 64) + b1) @ w2.view(64, 64) + b2) @ w3 + b3
    ((y - t) ** 2).mean().backward()
    g = th.grad
    return {"theta": (th - 1e-3 * g / (g.abs() + 1e-8)).detach()}


def _exact_mesh(case, seed):
    v, tri = _mesh(case, seed)
    lo, hi = v[tri.ravel()].min(0), v[tri.ravel()].max(0)
    ext = hi - lo
    lo2, hi2 = lo - ext * np.float32(0.1), hi + ext * np.float32(0.1)
    w = hi2 - lo2
    res = int(np.ceil(w[0] / np.float32(case["dx"])))
    cell = w[0] / np.float32(res)
    nodes = [res + 1, int(np.ceil(np.float32(res) * w[1] / w[0])) + 1, int(np.ceil(np.float32(res) * w[2] / w[0])) + 1]
    dev = _dev()
    at = [torch.tensor((np.float32(lo2[k]) + np.float32(cell) * np.arange(nodes[k], dtype=np.float32)), device=dev).double()
          for k in range(3)]
    z, y, x = torch.meshgrid(at[2], at[1], at[0], indexing="ij")
    p = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)
    T = torch.tensor(v[tri], device=dev).double()
    a, b, c = T[:, 0], T[:, 1], T[:, 2]
    mid = torch.tensor((lo + hi) * np.float32(0.5), device=dev).double()
    nor = torch.linalg.cross(b - a, a - c)
    out = []
    for q in p.split(2048):
        d2, side = None, 0
        for o, e in ((a, b - a), (b, c - b), (c, a - c)):
            r = q[:, None] - o
            side = side + torch.sign((r * torch.linalg.cross(e, nor)).sum(-1))
            k = ((r * e).sum(-1) / (e * e).sum(-1)).clamp(_f(1e-4), 1.0)
            l2 = ((k[..., None] * e - r) ** 2).sum(-1)
            d2 = l2 if d2 is None else torch.minimum(d2, l2)
        flat = ((q[:, None] - a) * nor).sum(-1) ** 2 / (nor * nor).sum(-1)
        dist = torch.where(side < 2, d2, flat).min(1).values.sqrt().clamp_min(1e-5)
        # crossings of the ray to the middle of the bounds and beyond
        dr = (mid - q) / (mid - q).norm(dim=1, keepdim=True)
        h = torch.linalg.cross(dr[:, None].expand(-1, len(a), -1), (c - a).expand(len(q), -1, -1))
        det = (h * (b - a)).sum(-1)
        s = q[:, None] - a
        u = (s * h).sum(-1) / det
        k = torch.linalg.cross(s, (b - a).expand(len(q), -1, -1))
        w_ = (dr[:, None] * k).sum(-1) / det
        t = (k * (c - a)).sum(-1) / det
        hits = ((u >= 0) & (w_ >= 0) & (u + w_ <= 1) & (t > 0)).sum(1)
        out.append(torch.where(hits % 2 == 1, -dist, dist))
    return {"nodes": None, "origin": None, "spacing": None, "values": torch.cat(out), "stuck": None}


def _grid_bounds(case):
    """UtilBuildGridForDomain: an even number of cells of 2 x spacing about the box's centre."""
    box = np.asarray(_box(case), np.float64)
    lo, hi = np.float32(-box / 2), np.float32(box / 2)
    length = np.float32(case["spacing"]) * np.float32(2.0)
    m = np.ceil(np.abs(hi - lo) * (np.float32(1) / length)).astype(np.int32)
    half = m.astype(np.float32) * np.float32(0.5 * float(length))
    mid = (lo + hi) * np.float32(0.5)
    return mid - half, mid + half


def _exact_surface(case, seed):
    pos, _, _ = _single(case, seed)
    x = pos.double()
    lo, hi = _grid_bounds(case)
    ds = np.float32(case["spacing"]) * np.float32(2.0)
    nodes = [int(np.ceil((hi[k] - lo[k]) / ds)) + 1 for k in range(3)]
    R = _f(2 * case["spacing"])
    far = float(np.sqrt(((hi - lo).astype(np.float64) ** 2).sum()))
    at = [torch.tensor(np.float32(lo[k] + ds * np.float32(0.5)) + ds * np.arange(nodes[k], dtype=np.float32),
                       device=x.device).double() for k in range(3)]
    out = []
    for zc in at[2].split(16):
        z, y, xx = torch.meshgrid(zc, at[1], at[0], indexing="ij")
        q = torch.stack([xx.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)
        i, j = _near(x, q, R)
        w = (1 - ((q[i] - x[j]) ** 2).sum(1) / (R * R)) ** 3
        tot = torch.zeros(len(q), device=x.device, dtype=torch.float64).index_add_(0, i, w)
        c = torch.zeros_like(q).index_add_(0, i, x[j] * w[:, None]) / tot[:, None]
        ok = (tot > 0) & torch.stack([q[:, k] <= float(hi[k]) for k in range(3)]).all(0)
        out.append(torch.where(ok, (q - c).norm(dim=1) - 0.25 * R, torch.full_like(tot, far)))
    return {"nodes": None, "values": torch.cat(out), "points": None, "normals": None, "triangles": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "advance", "batch", "learned"):
        return _exact_step(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "mesh":
        return _exact_mesh(case, seed)
    if kind == "surface":
        return _exact_surface(case, seed)
    if kind == "frame":
        pos, vel, _ = _single(case, seed)
        read = lambda a: np.array(["%g" % z for z in a.double().cpu().numpy().ravel()], "f8").reshape(-1, 3)  # noqa: E731
        return {"text": None, "pos": read(pos), "vel": read(vel)}
    return None
