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
// A node's candidates (216 in a full block) are tested four at a time, by squared distance against
// the largest square whose root is below the radius, and the slots of those that count kept in shared
// memory in walk order; the weights then run over them alone.  With the weight in the walk, one
// load at a time and half the lanes idle, the pass waited for its loads at 38 % of the issue slots: 68 -> 45 us
// (129,168 nodes).  Blocks of 64, since most nodes of a field lie outside the fluid and end at once.
#include "bbg_internal.cuh"
#include "bbg_kernels.h"

namespace bbg {

namespace {

__device__ __forceinline__ float dist3(v3 a, float4 b) {
    const float ex = fs(a.x, b.x), ey = fs(a.y, b.y), ez = fs(a.z, b.z);
    return __fsqrt_rn(fa(fa(fm(ex, ex), fm(ey, ey)), fm(ez, ez)));
}

constexpr int kFieldThreads = 64, kFieldSlots = 64;   // slots kept before they are summed

__global__ void __launch_bounds__(kFieldThreads)
k_particle_sdf(SurfaceArgs A, float *__restrict__ out) {
    __shared__ unsigned near[kFieldSlots][kFieldThreads];
    const int t = threadIdx.x;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)A.nodes[0] * A.nodes[1] * A.nodes[2];
    if (i >= total) return;
    // DimensionalIndex and FieldGrid3f::GetDataPosition (vertex centred)
    const unsigned ux = (unsigned)(i % A.nodes[0]);
    const unsigned uy = (unsigned)((i / A.nodes[0]) % A.nodes[1]);
    const unsigned uz = (unsigned)(i / ((long long)A.nodes[0] * A.nodes[1]));
    const v3 p = V(fa(A.org[0], fm(A.sp[0], (float)ux)), fa(A.org[1], fm(A.sp[1], (float)uy)),
                   fa(A.org[2], fm(A.sp[2], (float)uz)));
    const GridDev &g = A.g;
    if (!inside3(p, V(g.bmin[0], g.bmin[1], g.bmin[2]), V(g.bmax[0], g.bmax[1], g.bmax[2]), A.iz6)) {
        out[i] = A.inf;
        return;
    }
    unsigned bad = 0;
    const unsigned c = grid_hash(g, make_float4(p.x, p.y, p.z, 0.f), A.iz, &bad);
    const int cx = (int)(c % (unsigned)g.nx), cy = (int)((c / (unsigned)g.nx) % (unsigned)g.ny);
    const int cz = (int)(c / ((unsigned)g.nx * (unsigned)g.ny));
    const float R = A.radius;
    float wsum = 0.f, ax = 0.f, ay = 0.f, az = 0.f;
    auto add = [&](unsigned s, float4 xi) {
        const float d = dist3(p, xi);
        if (A.method == 0) {
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
    for (int y = max(cy - 1, 0); y <= min(cy + 1, g.ny - 1); y++)
        for (int x = max(cx - 1, 0); x <= min(cx + 1, g.nx - 1); x++) {
            const unsigned row = (unsigned)x + (unsigned)y * g.nx;
            unsigned b[3], e[3];
#pragma unroll
            for (int z = 0; z < 3; z++) {
                const unsigned nb = row + min(z0 + z, z1) * plane;
                b[z] = __ldg(&A.start[nb]);
                e[z] = z0 + z <= z1 ? __ldg(&A.start[nb + 1]) : b[z];
            }
#pragma unroll
            for (int z = 0; z < 3; z++)
                for (unsigned s = b[z]; s < e[z]; s += 4) {
                    float4 xi[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) xi[u] = __ldg(&A.pos[min(s + u, e[z] - 1u)]);
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const float ex = fs(p.x, xi[u].x), ey = fs(p.y, xi[u].y), ez = fs(p.z, xi[u].z);
                        const float d2 = fa(fa(fm(ex, ex), fm(ey, ey)), fm(ez, ez));
                        near[kept][t] = s + u;
                        kept += s + u < e[z] && (A.method != 0 || d2 <= A.near2) ? 1 : 0;
                    }
                    if (kept > kFieldSlots - 5) flush();
                }
        }
    flush();
    if (A.method != 0) {
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
    k_particle_sdf<<<(unsigned)((total + kFieldThreads - 1) / kFieldThreads), kFieldThreads, 0, s>>>(A, out);
}

}  // namespace bbg
