// surface.cu -- the surface app's particle-to-field step (apps/surface.cpp:276-470,
// ParticlesToSDF_Surface with ZhuBridsonSDF or SphSDF) on the sorted grid.
//
// One thread per node of the vertex-centred field: the node's position, the domain test,
// the hashed cell and its 27 neighbours in the reference's order (y, then x, then z), each
// cell's particles in chain order (the slot range of the last distribution).  Every float
// operation is explicitly rounded in the reference's order; the steps the reference takes
// in double (the cubic weight of Zhu-Bridson, the std kernel's constant) give the double's result
// (double_cube): 262,144 particles, 111 -> 70 us.
//
// Zhu-Bridson: a node's candidates (216 in a full block) are tested four at a time, by squared
// distance against the largest square whose root is below the radius, and the slots of those that count
// kept in shared memory in walk order; the weights then run over them alone.  With the weight in the
// walk, one load at a time and half the lanes idle, the pass waited for its loads at 38 % of the issue
// slots: 68 -> 45 us (129,168 nodes).  The lanes of a warp walk together and sum their lists up together,
// before a column that one of them may have no room for: lists summed up whenever a lane's was full took
// the other lanes' time as well (fields of 59,319 nodes, the whole call: a radius of two cells 174 -> 109
// us, particles at twice the rest density 209 -> 97).  64 slots: 48 are as good but for
// dense particles (two cells' radius 171 -> 298 us).  SPH: every candidate counts, so the weights
// stay in the walk, four loads at a time (208 -> 86 us; with lists in between 208).
// Blocks of 64, since most nodes of a field lie outside the fluid and end at once.
#include "bbg_internal.cuh"
#include "bbg_kernels.h"

namespace bbg {

namespace {

__device__ __forceinline__ float dist3(v3 a, float4 b) {
    const float ex = fs(a.x, b.x), ey = fs(a.y, b.y), ez = fs(a.z, b.z);
    return __fsqrt_rn(fa(fa(fm(ex, ex), fm(ey, ey)), fm(ez, ez)));
}

constexpr int kFieldThreads = 64, kFieldSlots = 64;   // slots kept before they are summed

// ZHU: the Zhu-Bridson field, else the SPH one
template <bool ZHU>
__global__ void __launch_bounds__(kFieldThreads)
k_particle_sdf(SurfaceArgs A, float *__restrict__ out) {
    __shared__ unsigned near[ZHU ? kFieldSlots : 1][kFieldThreads];
    constexpr unsigned full = 0xffffffffu;
    const int t = threadIdx.x;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)A.nodes[0] * A.nodes[1] * A.nodes[2];
    // DimensionalIndex and FieldGrid3f::GetDataPosition (vertex centred)
    const unsigned ux = (unsigned)(i % A.nodes[0]);
    const unsigned uy = (unsigned)((i / A.nodes[0]) % A.nodes[1]);
    const unsigned uz = (unsigned)(i / ((long long)A.nodes[0] * A.nodes[1]));
    const v3 p = V(fa(A.org[0], fm(A.sp[0], (float)ux)), fa(A.org[1], fm(A.sp[1], (float)uy)),
                   fa(A.org[2], fm(A.sp[2], (float)uz)));
    const GridDev &g = A.g;
    const bool in = i < total &&
                    inside3(p, V(g.bmin[0], g.bmin[1], g.bmin[2]), V(g.bmax[0], g.bmax[1], g.bmax[2]), A.iz6);
    if (i < total && !in) out[i] = A.inf;
    if (!__any_sync(full, in)) return;
    unsigned bad = 0;
    const unsigned c = grid_hash(g, make_float4(p.x, p.y, p.z, 0.f), A.iz, &bad);
    const int cx = (int)(c % (unsigned)g.nx), cy = (int)((c / (unsigned)g.nx) % (unsigned)g.ny);
    const int cz = (int)(c / ((unsigned)g.nx * (unsigned)g.ny));
    const float R = A.radius;
    float wsum = 0.f, ax = 0.f, ay = 0.f, az = 0.f;
    auto add = [&](unsigned s, float4 xi) {
        const float d = dist3(p, xi);
        if (ZHU) {
            // ZhuBridsonSDF: k_cub(|p - x| / R) = Max(0, (1 - s^2)^3), the cube in double
            if (d < R) {
                const float t = fdv(d, R);
                const float cub = double_cube_1m(fm(t, t));
                const float w = 0.f < cub ? cub : 0.f;
                wsum = fa(wsum, w);
                ax = fa(ax, fm(xi.x, w));
                ay = fa(ay, fm(xi.y, w));
                az = fa(az, fm(xi.z, w));
            }
        } else {
            // SphSDF: (mass / rho) W_std(d) at radius R (kernel.cpp:123-132)
            const float d2 = fm(d, d);
            const float of = fs(d2, A.r2);
            float w = 0.f;
            if (!(fabsf(of) < A.iz || of > 0.f)) {
                w = double_cube(A.wc, A.wh, A.wl, fs(1.f, fdv(d2, A.r2)));
            }
            wsum = fa(wsum, fm(fdv(A.mass, A.rho[s]), w));
        }
    };
    int kept = 0;
    auto flush = [&]() {
        for (int q = 0; q < kept; q += 4) {
            unsigned s[4];
            float4 x[4];
#pragma unroll
            for (int u = 0; u < 4; u++) s[u] = near[min(q + u, kept - 1)][t];
#pragma unroll
            for (int u = 0; u < 4; u++) x[u] = __ldg(&A.pos[s[u]]);
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (q + u < kept) add(s[u], x[u]);
        }
        kept = 0;
    };
    const unsigned plane = (unsigned)g.nx * (unsigned)g.ny;
    const unsigned z0 = (unsigned)max(cz - 1, 0), z1 = (unsigned)min(cz + 1, g.nz - 1);
    // the warp's lanes go through the nine columns of the 27 cells together
    // (a column's ranges are requested a column ahead)
    unsigned nb[3], ne[3];
    auto ranges = [&](int q) {
        const int y = cy - 1 + q / 3, x = cx - 1 + q % 3;
        const bool column = in && y >= 0 && y < g.ny && x >= 0 && x < g.nx;
        const unsigned row = (unsigned)x + (unsigned)y * g.nx;
#pragma unroll
        for (int z = 0; z < 3; z++) {
            nb[z] = ne[z] = 0;
            if (column && z0 + z <= z1) {
                const unsigned cell = row + (z0 + z) * plane;
                nb[z] = __ldg(&A.start[cell]);
                ne[z] = __ldg(&A.start[cell + 1]);
            }
        }
    };
    ranges(0);
#pragma unroll 1
    for (int q = 0; q < 9; q++) {
        unsigned b[3], e[3];
#pragma unroll
        for (int z = 0; z < 3; z++) {
            b[z] = nb[z];
            e[z] = ne[z];
        }
        if (q < 8) ranges(q + 1);
        const unsigned n0 = e[0] - b[0], n1 = n0 + (e[1] - b[1]), n = n1 + (e[2] - b[2]);
        const unsigned most = __reduce_max_sync(full, n);
        if (most == 0) continue;
        // room for the column in each lane's list, or all lanes sum theirs up together
        if (ZHU && __any_sync(full, kept + (int)min(n, 1u << 20) > kFieldSlots - 4)) flush();
        auto take = [&](unsigned s, bool valid, float4 xi) {
            if (ZHU) {
                const float ex = fs(p.x, xi.x), ey = fs(p.y, xi.y), ez = fs(p.z, xi.z);
                const float d2 = fa(fa(fm(ex, ex), fm(ey, ey)), fm(ez, ez));
                near[kept][t] = s;
                kept += valid && d2 <= A.near2 ? 1 : 0;
            } else if (valid) {
                add(s, xi);
            }
        };
        if (most <= 4) {   // scattered particles: the column at once (1.5 M nodes 155 -> 141 us)
            unsigned s[4];
            float4 xi[4];
#pragma unroll
            for (unsigned u = 0; u < 4; u++) s[u] = u < n0 ? b[0] + u : u < n1 ? b[1] + (u - n0) : u < n ? b[2] + (u - n1) : 0u;
#pragma unroll
            for (int u = 0; u < 4; u++) xi[u] = __ldg(&A.pos[s[u]]);
#pragma unroll
            for (unsigned u = 0; u < 4; u++) take(s[u], u < n, xi[u]);
            continue;
        }
#pragma unroll
        for (int z = 0; z < 3; z++)
            for (unsigned s = b[z]; s < e[z]; s += 4) {
                if (ZHU && kept > kFieldSlots - 4) flush();   // a column of more than the list
                float4 xi[4];
#pragma unroll
                for (int u = 0; u < 4; u++) xi[u] = __ldg(&A.pos[min(s + u, e[z] - 1u)]);
#pragma unroll
                for (int u = 0; u < 4; u++) take(s + u, s + u < e[z], xi[u]);
            }
    }
    if (ZHU) flush();
    if (!in) return;
    if (!ZHU) {
        out[i] = fs(0.5f, wsum);
    } else if (wsum > 0.f) {
        const float inv = __double2float_rn(__ddiv_rn(1.0, (double)wsum));
        const float4 m = make_float4(fm(ax, inv), fm(ay, inv), fm(az, inv), 0.f);
        out[i] = fs(dist3(p, m), A.offset);
    } else {
        out[i] = A.inf;
    }
}

}  // namespace

void launch_particle_sdf(const SurfaceArgs &A, float *out, cudaStream_t s) {
    const long long total = (long long)A.nodes[0] * A.nodes[1] * A.nodes[2];
    const unsigned blocks = (unsigned)((total + kFieldThreads - 1) / kFieldThreads);
    if (A.method == 0) k_particle_sdf<true><<<blocks, kFieldThreads, 0, s>>>(A, out);
    else k_particle_sdf<false><<<blocks, kFieldThreads, 0, s>>>(A, out);
}

}  // namespace bbg
