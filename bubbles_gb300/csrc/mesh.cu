// mesh.cu -- the signed-distance field of a triangle mesh on the device: GenerateShapeSDF of
// a mesh shape (src/core/shape.cpp:409-424, 479-510).
//
// One thread per grid node.  The distance is the least DistanceTriangle over the triangles
// (src/shapes/bvh.cpp:212-242; the reference's BVH only prunes, the minimum is the same
// value); the sign comes from MeshIsPointInside (shape.cpp:349-369): a ray from the node
// towards the mesh bounds' centre, the closest hit found (IntersectTriangle, bvh.cpp:244-
// 373, a watertight ray-triangle test with floating-point error bounds), the ray re-spawned
// past it (SpawnRayInDirection / OffsetRayOrigin, interaction.h:51-55, geometry.h:1843-
// 1858), hits counted until none is left; odd means inside.  Every operation is an
// explicitly rounded float or double operation in the reference's order, so the node values
// are the reference's except where two triangles tie for the closest hit (the reference's
// BVH order picks one of them, here the last by index does).  Triangles are read by all
// threads of a warp together (broadcast loads through L1).
//
// FP64 runs at 1/64 of the FP32 rate here, so nothing of a triangle alone is computed per node:
// k_mesh_records does the reference's double cross products once a triangle, and the
// double comparisons with constants are float comparisons with the least float above them.
#include "bbg_internal.cuh"
#include "bbg_kernels.h"

#include <algorithm>
#include <utility>
#include <vector>

namespace bbg {

static inline int blocks_for(long long n, int t) { return (int)((n + t - 1) / t); }

namespace {

__device__ __forceinline__ float sgn(float a) { return a > 0.f ? 1.f : (a < 0.f ? -1.f : 0.f); }

// Cross in double, rounded to float per component (geometry.h:906-914)
__device__ __forceinline__ v3 cross_d(v3 a, v3 b) {
    const double ax = a.x, ay = a.y, az = a.z, bx = b.x, by = b.y, bz = b.z;
    return V(__double2float_rn(__dsub_rn(__dmul_rn(ay, bz), __dmul_rn(az, by))),
             __double2float_rn(__dsub_rn(__dmul_rn(az, bx), __dmul_rn(ax, bz))),
             __double2float_rn(__dsub_rn(__dmul_rn(ax, by), __dmul_rn(ay, bx))));
}

// Clamp(v, 0.0001, 1.0) with the double bounds returned as floats; below: the least float
// that is not below 0.0001
__device__ __forceinline__ float clamp_edge(float v, float below) {
    if (v < below) return 0.0001f;
    if (v > 1.f) return 1.f;
    return v;
}

// What DistanceTriangle (bvh.cpp:212-242) takes from the triangle alone, in 9 float4
struct TriDist {
    v3 a, b, c, ba, cb, ac, nor, n0, n1, n2;   // n0 = Cross(ba, nor) and so on
    float l0, l1, l2, ln;                      // |ba|^2, |cb|^2, |ac|^2, |nor|^2
};
constexpr int kDistRec = 36, kRayRec = 12;   // floats per triangle (34 and 9 used)

__device__ __forceinline__ TriDist load_dist(const float4 *__restrict__ r) {
    const float4 q0 = __ldg(r), q1 = __ldg(r + 1), q2 = __ldg(r + 2), q3 = __ldg(r + 3), q4 = __ldg(r + 4);
    const float4 q5 = __ldg(r + 5), q6 = __ldg(r + 6), q7 = __ldg(r + 7), q8 = __ldg(r + 8);
    TriDist t;
    t.a = V(q0.x, q0.y, q0.z); t.b = V(q0.w, q1.x, q1.y); t.c = V(q1.z, q1.w, q2.x);
    t.ba = V(q2.y, q2.z, q2.w); t.cb = V(q3.x, q3.y, q3.z); t.ac = V(q3.w, q4.x, q4.y);
    t.nor = V(q4.z, q4.w, q5.x); t.n0 = V(q5.y, q5.z, q5.w); t.n1 = V(q6.x, q6.y, q6.z);
    t.n2 = V(q6.w, q7.x, q7.y);
    t.l0 = q7.z; t.l1 = q7.w; t.l2 = q8.x; t.ln = q8.y;
    return t;
}

// The squared DistanceTriangle: the reference's value is its square root, which keeps order, so
// the least one is rooted once.
__device__ __forceinline__ float distance_triangle2(v3 p, const TriDist &t, float below) {
    const v3 pa = vsub(p, t.a), pb = vsub(p, t.b), pc = vsub(p, t.c);
    const float s = fa(fa(sgn(vdot(t.n0, pa)), sgn(vdot(t.n1, pb))), sgn(vdot(t.n2, pc)));
    if (s < 2.f) {
        const float e0 = vlen2(vsub(vmul(t.ba, clamp_edge(fdv(vdot(t.ba, pa), t.l0), below)), pa));
        const float e1 = vlen2(vsub(vmul(t.cb, clamp_edge(fdv(vdot(t.cb, pb), t.l1), below)), pb));
        const float e2 = vlen2(vsub(vmul(t.ac, clamp_edge(fdv(vdot(t.ac, pc), t.l2), below)), pc));
        return rmin(rmin(e0, e1), e2);
    }
    const float d = vdot(t.nor, pa);
    return fdv(fm(d, d), t.ln);
}

// The records of every triangle: corners for the ray passes (the caller's order), TriDist for
// the distance pass (the Morton-ordered copy).
__global__ void k_mesh_records(const float *__restrict__ tri, const float *__restrict__ dtri, int ntri,
                               float *__restrict__ ray, float *__restrict__ dist) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntri) return;
    for (int k = 0; k < 9; k++) ray[kRayRec * (size_t)t + k] = tri[9 * (size_t)t + k];
    const float *q = dtri + 9 * (size_t)t;
    const v3 a = V(q[0], q[1], q[2]), b = V(q[3], q[4], q[5]), c = V(q[6], q[7], q[8]);
    const v3 ba = vsub(b, a), cb = vsub(c, b), ac = vsub(a, c);
    const v3 nor = cross_d(ba, ac);
    const v3 v[10] = {a, b, c, ba, cb, ac, nor, cross_d(ba, nor), cross_d(cb, nor), cross_d(ac, nor)};
    float *o = dist + kDistRec * (size_t)t;
    for (int k = 0; k < 10; k++) {
        o[3 * k] = v[k].x;
        o[3 * k + 1] = v[k].y;
        o[3 * k + 2] = v[k].z;
    }
    o[30] = vlen2(ba);
    o[31] = vlen2(cb);
    o[32] = vlen2(ac);
    o[33] = vlen2(nor);
    o[34] = o[35] = 0.f;
}

__device__ __forceinline__ float comp(v3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }
__device__ __forceinline__ v3 permute(v3 v, int x, int y, int z) { return V(comp(v, x), comp(v, y), comp(v, z)); }
__device__ __forceinline__ float max3abs(float a, float b, float c) {   // MaxComponent(Abs(v))
    return rmax(fabsf(a), rmax(fabsf(b), fabsf(c)));
}

// error-bound factors, and the least floats not below 1e-8 and 0.0001 (double comparisons)
struct Gammas { float g2, g3, g5, g7, zero, edge; };

// A direction with what IntersectTriangle and Bounds3::Intersect take from it alone
struct RayDir {
    v3 dir, inv;          // 1 / dir
    float sx, sy, sz;     // shear to the frame whose z is dir's largest axis
    int kx, ky, kz;
};
__device__ __forceinline__ RayDir ray_dir(v3 dir) {
    RayDir r;
    r.dir = dir;
    r.inv = V(fdv(1.f, dir.x), fdv(1.f, dir.y), fdv(1.f, dir.z));
    const v3 ad = V(fabsf(dir.x), fabsf(dir.y), fabsf(dir.z));
    r.kz = (ad.x > ad.y) ? ((ad.x > ad.z) ? 0 : 2) : ((ad.y > ad.z) ? 1 : 2);
    r.kx = r.kz == 2 ? 0 : r.kz + 1;
    r.ky = r.kx == 2 ? 0 : r.kx + 1;
    const v3 d = permute(dir, r.kx, r.ky, r.kz);
    r.sx = fdv(-d.x, d.z);
    r.sy = fdv(-d.y, d.z);
    r.sz = fdv(1.f, d.z);
    return r;
}

struct Hit { v3 p, err, n; float t; };

// a b - c d in double, for edge functions near zero.  Out of line: inlined, the compiler evaluates
// it for every triangle and selects.
static __device__ __noinline__ float edge_exact(float a, float b, float c, float d) {
    return __double2float_rn(__dsub_rn(__dmul_rn((double)a, (double)b), __dmul_rn((double)c, (double)d)));
}

// IntersectTriangle (bvh.cpp:244-373) against a ray with tMax; on a hit, tmax and hit
// are updated.
__device__ __forceinline__ bool intersect_triangle(v3 o, const RayDir &R, float &tmax, v3 p0, v3 p1, v3 p2,
                                                   const Gammas &G, Hit &hit) {
    const float sx = R.sx, sy = R.sy, sz = R.sz;
    v3 p0t = permute(vsub(p0, o), R.kx, R.ky, R.kz);
    v3 p1t = permute(vsub(p1, o), R.kx, R.ky, R.kz);
    v3 p2t = permute(vsub(p2, o), R.kx, R.ky, R.kz);
    p0t.x = fa(p0t.x, fm(sx, p0t.z));
    p0t.y = fa(p0t.y, fm(sy, p0t.z));
    p1t.x = fa(p1t.x, fm(sx, p1t.z));
    p1t.y = fa(p1t.y, fm(sy, p1t.z));
    p2t.x = fa(p2t.x, fm(sx, p2t.z));
    p2t.y = fa(p2t.y, fm(sy, p2t.z));
    float e0 = fs(fm(p1t.x, p2t.y), fm(p1t.y, p2t.x));
    float e1 = fs(fm(p2t.x, p0t.y), fm(p2t.y, p0t.x));
    float e2 = fs(fm(p0t.x, p1t.y), fm(p0t.y, p1t.x));
    if (fabsf(e0) < G.zero || fabsf(e1) < G.zero || fabsf(e2) < G.zero) {
        e0 = edge_exact(p2t.y, p1t.x, p2t.x, p1t.y);
        e1 = edge_exact(p0t.y, p2t.x, p0t.x, p2t.y);
        e2 = edge_exact(p1t.y, p0t.x, p1t.x, p0t.y);
    }
    if ((e0 < 0.f || e1 < 0.f || e2 < 0.f) && (e0 > 0.f || e1 > 0.f || e2 > 0.f)) return false;
    const float det = fa(fa(e0, e1), e2);
    if (fabsf(det) < G.zero) return false;
    p0t.z = fm(p0t.z, sz);
    p1t.z = fm(p1t.z, sz);
    p2t.z = fm(p2t.z, sz);
    const float ts = fa(fa(fm(e0, p0t.z), fm(e1, p1t.z)), fm(e2, p2t.z));
    if (det < 0.f && (ts >= 0.f || ts < fm(tmax, det))) return false;
    if (det > 0.f && (ts <= 0.f || ts > fm(tmax, det))) return false;
    const float inv = fdv(1.f, det);
    const float b0 = fm(e0, inv), b1 = fm(e1, inv), b2 = fm(e2, inv);
    const float t = fm(ts, inv);
    const float maxzt = max3abs(p0t.z, p1t.z, p2t.z);
    const float dz = fm(G.g3, maxzt);
    const float maxxt = max3abs(p0t.x, p1t.x, p2t.x);
    const float maxyt = max3abs(p0t.y, p1t.y, p2t.y);
    const float dx = fm(G.g5, fa(maxxt, maxzt));
    const float dy = fm(G.g5, fa(maxyt, maxzt));
    const float de = fm(2.f, fa(fa(fm(fm(G.g2, maxxt), maxyt), fm(dy, maxxt)), fm(dx, maxyt)));
    const float maxe = max3abs(e0, e1, e2);
    const float dt = fm(fm(3.f, fa(fa(fm(fm(G.g3, maxe), maxzt), fm(de, maxzt)), fm(dz, maxe))), fabsf(inv));
    if (t <= dt) return false;
    const float xs = fa(fa(fabsf(fm(b0, p0.x)), fabsf(fm(b1, p1.x))), fabsf(fm(b2, p2.x)));
    const float ys = fa(fa(fabsf(fm(b0, p0.y)), fabsf(fm(b1, p1.y))), fabsf(fm(b2, p2.y)));
    const float zs = fa(fa(fabsf(fm(b0, p0.z)), fabsf(fm(b1, p1.z))), fabsf(fm(b2, p2.z)));
    hit.err = vmul(V(xs, ys, zs), G.g7);
    hit.p = vadd(vadd(vmul(p0, b0), vmul(p1, b1)), vmul(p2, b2));
    const v3 nn = cross_d(vsub(p0, p2), vsub(p1, p2));
    hit.n = vdiv(nn, vlen(nn));
    hit.t = t;
    tmax = t;
    return true;
}

// Bounds3::Intersect (geometry.h:1881-1898)
__device__ __forceinline__ bool hits_bounds(v3 lo, v3 hi, v3 o, v3 inv, float tmax, float g3) {
    float t0 = 0.f, t1 = tmax;
    const float grow = fa(1.f, fm(2.f, g3));
#pragma unroll
    for (int k = 0; k < 3; k++) {
        float tn = fm(fs(comp(lo, k), comp(o, k)), comp(inv, k));
        float tf = fm(fs(comp(hi, k), comp(o, k)), comp(inv, k));
        if (tn > tf) {
            const float x = tn;
            tn = tf;
            tf = x;
        }
        tf = fm(tf, grow);
        t0 = tn > t0 ? tn : t0;
        t1 = tf < t1 ? tf : t1;
        if (t0 > t1) return false;
    }
    return true;
}

__device__ __forceinline__ float next_up(float v) {
    if (isinf(v) && v > 0.f) return v;
    if (v == -0.f) v = 0.f;
    unsigned u = __float_as_uint(v);
    u = v >= 0.f ? u + 1u : u - 1u;
    return __uint_as_float(u);
}

__device__ __forceinline__ float next_down(float v) {
    if (isinf(v) && v < 0.f) return v;
    if (v == 0.f) v = -0.f;
    unsigned u = __float_as_uint(v);
    u = v > 0.f ? u - 1u : u + 1u;
    return __uint_as_float(u);
}

// OffsetRayOrigin (geometry.h:1843-1858): past the hit by the error bound + 0.0001 along n
__device__ v3 offset_origin(const Hit &h, v3 w) {
    const float d = __double2float_rn((double)vdot(V(fabsf(h.n.x), fabsf(h.n.y), fabsf(h.n.z)), h.err) + 0.0001);
    v3 off = vmul(h.n, d);
    if (vdot(w, h.n) < 0.f) off = V(-off.x, -off.y, -off.z);
    v3 po = vadd(h.p, off);
    po.x = off.x > 0.f ? next_up(po.x) : (off.x < 0.f ? next_down(po.x) : po.x);
    po.y = off.y > 0.f ? next_up(po.y) : (off.y < 0.f ? next_down(po.y) : po.y);
    po.z = off.z > 0.f ? next_up(po.z) : (off.z < 0.f ? next_down(po.z) : po.z);
    return po;
}

constexpr int kMaxRayHits = 256;   // a ray stuck on degenerate geometry gives up (outside)

// Triangles are visited in tiles of kMeshTile consecutive triangles, each split into
// kMeshTile / kMeshSub sub-tiles, every tile and sub-tile with its bounding box: one is
// skipped when its box cannot hold a better answer, which leaves every result equal to the
// scan over all triangles.
//  - distance: skipped when the box lies farther than the best distance so far by more than
//    1 % plus an absolute margin (1e-3 of the mesh's bounding diagonal), so a skipped
//    triangle's computed distance cannot be below the best despite rounding;
//  - rays: skipped when the conservative ray-box test (Bounds3::IntersectP with the gamma
//    growth, the test of the reference's BVH) rejects the box for the current tMax, which
//    never rejects a box holding a hit at or before tMax.
constexpr int kMeshTile = 64;
// Sub-tiles of 4 leave fewer triangles for twice the box tests inside a kept tile: the torus below, the whole
// call, 1,270 -> 1,091 us against 8 (of 2: 1,126; tiles of 32 with 4: 1,100, and twice the tiles to pass
// over in a large mesh).
constexpr int kMeshSub = 4;

// Boxes: 8 floats each, low corner then high corner.  Squared distance of p to a box:
__device__ __forceinline__ float box_distance2(const float4 *__restrict__ bx, v3 p) {
    const float4 l = __ldg(bx), h = __ldg(bx + 1);
    const float ex = fmaxf(fmaxf(l.x - p.x, p.x - h.x), 0.f);
    const float ey = fmaxf(fmaxf(l.y - p.y, p.y - h.y), 0.f);
    const float ez = fmaxf(fmaxf(l.z - p.z, p.z - h.z), 0.f);
    return ex * ex + ey * ey + ez * ez;
}

__device__ __forceinline__ bool box_on_ray(const float4 *__restrict__ bx, v3 o, v3 inv, float tmax, float g3) {
    const float4 l = __ldg(bx), h = __ldg(bx + 1);
    return hits_bounds(V(l.x, l.y, l.z), V(h.x, h.y, h.z), o, inv, tmax, g3);
}

// f(t) for every triangle t of the tiles and sub-tiles that keep(box) accepts, in order
template <class Keep, class F>
__device__ __forceinline__ void mesh_walk(const float4 *__restrict__ tiles, int ntri, Keep &&keep, F &&f) {
    const int ntiles = (ntri + kMeshTile - 1) / kMeshTile, nsub = (ntri + kMeshSub - 1) / kMeshSub;
    const float4 *sub = tiles + 2 * ntiles;
    for (int b = 0; b < ntiles; b++) {
        if (!keep(tiles + 2 * b)) continue;
        const int s1 = min(nsub, (b + 1) * (kMeshTile / kMeshSub));
        for (int q = b * (kMeshTile / kMeshSub); q < s1; q++) {
            if (!keep(sub + 2 * q)) continue;
            const int t1 = min(ntri, (q + 1) * kMeshSub);
            for (int t = q * kMeshSub; t < t1; t++) f(t);
        }
    }
}

// Bound: FP32 issue slots of the triangle tests that the boxes leave.  The lanes of a warp share
// them when their nodes are near one another in all three directions: 22.7 of 32 lanes active a
// triangle with bricks, 12.9 with 32 nodes in a row.  Torus of 1,152 triangles, 0.43M nodes: 23.0
// ms with the double products per node, 1.49 ms without, 0.88 ms in bricks, 0.74 ms with sub-tiles of
// 4 (rays 0.35 of it before).
__global__ void __launch_bounds__(128)
k_mesh_sdf(const float4 *__restrict__ ray, int ntri, const float4 *__restrict__ tiles, const float4 *__restrict__ dist,
           const float4 *__restrict__ dtiles, float margin, SdfDev g, v3 lo, v3 hi, Gammas G, float *__restrict__ out,
           unsigned *__restrict__ stuck) {
    // a warp takes 4 x 4 x 2 nodes, a block 8 x 4 x 4
    const unsigned bx = ((unsigned)g.nx + 7u) / 8u, by = ((unsigned)g.ny + 3u) / 4u;
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const unsigned i = 8u * (blockIdx.x % bx) + 4u * (wid & 1u) + (lane & 3u);
    const unsigned j = 4u * (blockIdx.x / bx % by) + ((lane >> 2) & 3u);
    const unsigned k = 4u * (blockIdx.x / bx / by) + 2u * (wid >> 1) + (lane >> 4);
    if (i >= (unsigned)g.nx || j >= (unsigned)g.ny || k >= (unsigned)g.nz) return;
    const unsigned id = i + (unsigned)g.nx * (j + (unsigned)g.ny * k);
    const v3 p = V(fa(g.org[0], fm(g.sp[0], (float)i)), fa(g.org[1], fm(g.sp[1], (float)j)),
                   fa(g.org[2], fm(g.sp[2], (float)k)));
    // MeshClosestDistance: the least DistanceTriangle (strictly smaller replaces; the least
    // value does not depend on the order, so this pass walks the Morton-ordered copy, the
    // sub-tile whose box is nearest first: its distances leave little of the rest)
    float d = 3.1622776601683794e+18f;   // SqrtInfinity
    float q2 = __int_as_float(0x7f800000), reach2 = q2;   // least squared distance, and of a box that matters
    auto visit = [&](int t) {
        const float q = distance_triangle2(p, load_dist(dist + (kDistRec / 4) * (size_t)t), G.edge);
        if (q < q2) {
            q2 = q;
            const float r = sqrtf(q) * 1.01f + margin;
            reach2 = r * r * 1.0001f;
        }
    };
    {
        const int ntiles = (ntri + kMeshTile - 1) / kMeshTile, nsub = (ntri + kMeshSub - 1) / kMeshSub;
        const float4 *sub = dtiles + 2 * ntiles;
        int tile = 0, first = 0;
        float near2 = box_distance2(dtiles, p);
        for (int b = 1; b < ntiles; b++) {
            const float e = box_distance2(dtiles + 2 * b, p);
            if (e < near2) {
                near2 = e;
                tile = b;
            }
        }
        first = tile * (kMeshTile / kMeshSub);
        const int s1 = min(nsub, first + kMeshTile / kMeshSub);
        near2 = box_distance2(sub + 2 * first, p);
        for (int b = first + 1; b < s1; b++) {
            const float e = box_distance2(sub + 2 * b, p);
            if (e < near2) {
                near2 = e;
                first = b;
            }
        }
        for (int t = first * kMeshSub; t < min(ntri, (first + 1) * kMeshSub); t++) visit(t);
    }
    mesh_walk(dtiles, ntri, [&](const float4 *bx) { return !(box_distance2(bx, p) > reach2); }, visit);
    const float root = __fsqrt_rn(q2);
    if (root < d) d = root;
    // MeshIsPointInside: ray towards the bounds' centre, closest hits counted
    const v3 center = vmul(vadd(lo, hi), 0.5f);
    const v3 to = vsub(center, p);
    const RayDir R = ray_dir(vdiv(to, vlen(to)));
    v3 o = p;
    int hits = 0;
    bool done = false;
    for (int it = 0; it < kMaxRayHits && !done; it++) {
        float tmax = 3.402823466e+38f;   // Infinity
        Hit h;
        bool any = false;
        if (hits_bounds(lo, hi, o, R.inv, tmax, G.g3)) {
            mesh_walk(tiles, ntri, [&](const float4 *bx) { return box_on_ray(bx, o, R.inv, tmax, G.g3); }, [&](int t) {
                const float4 *q = ray + (kRayRec / 4) * (size_t)t;
                const float4 u = __ldg(q), v = __ldg(q + 1), w = __ldg(q + 2);
                any |= intersect_triangle(o, R, tmax, V(u.x, u.y, u.z), V(u.w, v.x, v.y), V(v.z, v.w, w.x), G, h);
            });
        }
        if (!any) {
            done = true;
        } else {
            hits++;
            o = offset_origin(h, R.dir);
        }
    }
    if (!done) {
        atomicAdd(stuck, 1u);
        hits = 0;
    }
    const bool interior = (hits % 2) != 0 && hits > 0;
    const float psd = rmax(fabsf(d), 0.00001f);
    out[id] = interior ? -psd : psd;
}

}  // namespace

// boxes of the tiles, then of the sub-tiles (8 floats each)
int mesh_tiles(int ntri) { return (ntri + kMeshTile - 1) / kMeshTile + (ntri + kMeshSub - 1) / kMeshSub; }

static void tile_boxes(const float *tri, int ntri, int size, float *tiles) {
    for (int b = 0; b < (ntri + size - 1) / size; b++) {
        float *bx = tiles + 8 * b;
        for (int k = 0; k < 3; k++) {
            bx[k] = 3.402823466e+38f;
            bx[4 + k] = -3.402823466e+38f;
        }
        bx[3] = bx[7] = 0.f;
        for (int t = b * size; t < ntri && t < (b + 1) * size; t++)
            for (int c = 0; c < 3; c++)
                for (int k = 0; k < 3; k++) {
                    const float x = tri[9 * (size_t)t + 3 * c + k];
                    bx[k] = x < bx[k] ? x : bx[k];
                    bx[4 + k] = x > bx[4 + k] ? x : bx[4 + k];
                }
    }
}

void mesh_tile_bounds(const float *tri, int ntri, float *tiles) {
    tile_boxes(tri, ntri, kMeshTile, tiles);
    tile_boxes(tri, ntri, kMeshSub, tiles + 8 * ((ntri + kMeshTile - 1) / kMeshTile));
}

// The triangles in the Morton order of their centroids (30-bit codes in the mesh bounds,
// ties by index), for the distance pass's tiles.
void mesh_morton_order(const float *tri, int ntri, const float lo[3], const float hi[3], float *sorted) {
    std::vector<std::pair<unsigned, int>> key((size_t)ntri);
    for (int t = 0; t < ntri; t++) {
        unsigned code = 0;
        unsigned q[3];
        for (int k = 0; k < 3; k++) {
            const float c = (tri[9 * (size_t)t + k] + tri[9 * (size_t)t + 3 + k] + tri[9 * (size_t)t + 6 + k]) / 3.f;
            const float ext = hi[k] - lo[k];
            float u = ext > 0.f ? (c - lo[k]) / ext : 0.f;
            u = u < 0.f ? 0.f : (u > 1.f ? 1.f : u);
            q[k] = (unsigned)(u * 1023.f);
        }
        for (int bit = 9; bit >= 0; bit--)
            for (int k = 0; k < 3; k++) code = (code << 1) | ((q[k] >> bit) & 1u);
        key[(size_t)t] = std::make_pair(code, t);
    }
    std::sort(key.begin(), key.end());
    for (int r = 0; r < ntri; r++)
        for (int q = 0; q < 9; q++) sorted[9 * (size_t)r + q] = tri[9 * (size_t)key[(size_t)r].second + q];
}

size_t mesh_record_floats(int ntri) { return (size_t)(kDistRec + kRayRec) * (size_t)ntri; }

void launch_mesh_sdf(const float *tri, int ntri, const float *tiles, const float *dtri, const float *dtiles,
                     float margin, const SdfDev &g, const float lo[3], const float hi[3], const float gamma[4],
                     const float least[2], float *records, float *out, unsigned *stuck, cudaStream_t s) {
    const long long bricks = (((long long)g.nx + 7) / 8) * (((long long)g.ny + 3) / 4) * (((long long)g.nz + 3) / 4);
    const Gammas G = {gamma[0], gamma[1], gamma[2], gamma[3], least[0], least[1]};
    v3 l, h;
    l.x = lo[0]; l.y = lo[1]; l.z = lo[2];
    h.x = hi[0]; h.y = hi[1]; h.z = hi[2];
    float *dist = records, *ray = records + (size_t)kDistRec * (size_t)ntri;
    k_mesh_records<<<blocks_for(ntri, 128), 128, 0, s>>>(tri, dtri, ntri, ray, dist);
    const auto quads = [](const float *p) { return reinterpret_cast<const float4 *>(p); };
    k_mesh_sdf<<<(unsigned)bricks, 128, 0, s>>>(quads(ray), ntri, quads(tiles), quads(dist), quads(dtiles), margin,
                                                      g, l, h, G, out, stuck);
}

}  // namespace bbg
