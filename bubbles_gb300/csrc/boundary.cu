// boundary.cu -- boundary classification of the particles on the sorted grid:
// src/boundaries/lnm.h (LNMBoundary with its fast, Xiaowei and Dilts L2 filters,
// LNMBoundarySingle, LNMBoundaryExtended), xiaowei.h and dilts.h.
//
// The reference walks its cells' chains; here a cell's particles are the slot range of the
// last grid distribution (the chain order).  Cell passes run one thread per cell and only
// write their own cell's level, reading levels that no pass of the same launch changes,
// so they equal the reference's sequential sweeps.  Particle passes run one thread per
// slot and write in the caller's order.  Every float operation of the two geometric tests
// is explicitly rounded in the reference's order, the kernel weights' double steps included.
#include "bbg_internal.cuh"
#include "bbg_kernels.h"

#include <algorithm>

namespace bbg {

static inline int blocks_for(long long n, int t) { return (int)((n + t - 1) / t); }

namespace {

__device__ __forceinline__ unsigned held(const unsigned *start, unsigned c) { return start[c + 1] - start[c]; }

__global__ void k_lnm_l1(GridDev g, const unsigned *__restrict__ start, int *__restrict__ level) {
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.total) return;
    level[c] = -1;
    if (held(start, c) < 1) return;
    const int x = (int)(c % (unsigned)g.nx), y = (int)((c / (unsigned)g.nx) % (unsigned)g.ny);
    const int z = (int)(c / ((unsigned)g.nx * (unsigned)g.ny));
    const int x0 = x > 0 ? x - 1 : 0, x1 = x + 1 < g.nx ? x + 1 : g.nx - 1;
    const int y0 = y > 0 ? y - 1 : 0, y1 = y + 1 < g.ny ? y + 1 : g.ny - 1;
    const int z0 = z > 0 ? z - 1 : 0, z1 = z + 1 < g.nz ? z + 1 : g.nz - 1;
    if ((x1 - x0 + 1) * (y1 - y0 + 1) * (z1 - z0 + 1) != 27) {   // GetNeighborsOf count
        level[c] = 1;
        return;
    }
    for (int k = z0; k <= z1; k++)
        for (int j = y0; j <= y1; j++)
            for (int i = x0; i <= x1; i++)
                if (held(start, (unsigned)i + (unsigned)j * g.nx + (unsigned)k * g.nx * g.ny) == 0) {
                    level[c] = 1;
                    return;
                }
}

__global__ void k_lnm_l2(GridDev g, const unsigned *__restrict__ start, int *__restrict__ level, int delta) {
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.total) return;
    if (held(start, c) < 1 || level[c] == 1) return;
    const int x = (int)(c % (unsigned)g.nx), y = (int)((c / (unsigned)g.nx) % (unsigned)g.ny);
    const int z = (int)(c / ((unsigned)g.nx * (unsigned)g.ny));
    for (int k = z > 0 ? z - 1 : 0; k <= (z + 1 < g.nz ? z + 1 : g.nz - 1); k++)
        for (int j = y > 0 ? y - 1 : 0; j <= (y + 1 < g.ny ? y + 1 : g.ny - 1); j++)
            for (int i = x > 0 ? x - 1 : 0; i <= (x + 1 < g.nx ? x + 1 : g.nx - 1); i++) {
                const unsigned nb = (unsigned)i + (unsigned)j * g.nx + (unsigned)k * g.nx * g.ny;
                // an L2 write never turns a cell into or out of L1, so the reads are stable
                if (level[nb] == 1 && held(start, nb) <= (unsigned)delta) {
                    level[c] = 2;
                    return;
                }
            }
}

__global__ void k_lnm_particles(int n, const unsigned *__restrict__ cell, const int *__restrict__ pid,
                                const int *__restrict__ level, int *__restrict__ out) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int L = level[cell[q] & ~kWide];
    out[pid[q]] = (L == 1 || L == 2) ? L : 0;
}

__device__ __forceinline__ void coords(const GridDev &g, unsigned c, int u[3]) {
    u[0] = (int)(c % (unsigned)g.nx);
    u[1] = (int)((c / (unsigned)g.nx) % (unsigned)g.ny);
    u[2] = (int)(c / ((unsigned)g.nx * (unsigned)g.ny));
}

__device__ __forceinline__ unsigned linear(const GridDev &g, int x, int y, int z) {
    return (unsigned)x + (unsigned)y * (unsigned)g.nx + (unsigned)z * (unsigned)g.nx * (unsigned)g.ny;
}

__device__ __forceinline__ bool on_border(const GridDev &g, const int u[3]) {
    return u[0] == 0 || u[1] == 0 || u[2] == 0 || u[0] == g.nx - 1 || u[1] == g.ny - 1 || u[2] == g.nz - 1 ||
           g.nx < 3 || g.ny < 3 || g.nz < 3;
}

// LNMBoundaryAreCoords1x1: distinct cells at most one step apart on every axis
__device__ __forceinline__ bool adjacent(const int a[3], const int b[3]) {
    const int dx = abs(a[0] - b[0]), dy = abs(a[1] - b[1]), dz = abs(a[2] - b[2]);
    return dx < 2 && dy < 2 && dz < 2 && dx + dy + dz > 0;
}

// LNMBoundarySingleKernel (lnm.h:167-238).  The 5x5x5 walk (y, then x, then z) stops at the
// first empty adjacent cell (L1) or the first adjacent cell holding at most delta particles
// that lies on the border (L2).  Without a stop every empty cell of the walk is a source and
// every adjacent cell holding 1..delta particles a candidate, and the cell is L2 when a
// candidate touches a source: with no empty cell adjacent to this one, the sources a
// candidate touches are exactly the empty cells adjacent to the candidate, all inside the walk.
__global__ void k_lnm_single(GridDev g, const unsigned *__restrict__ start, int *__restrict__ level, int delta) {
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.total) return;
    level[c] = -1;
    if (held(start, c) == 0) return;
    int u[3];
    coords(g, c, u);
    if (on_border(g, u)) {
        level[c] = 1;
        return;
    }
    for (int j = u[1] - 2; j <= u[1] + 2; j++) {
        if (j < 0 || j >= g.ny) continue;
        for (int i = u[0] - 2; i <= u[0] + 2; i++) {
            if (i < 0 || i >= g.nx) continue;
            for (int k = u[2] - 2; k <= u[2] + 2; k++) {
                if (k < 0 || k >= g.nz) continue;
                const int f[3] = {i, j, k};
                const unsigned fid = linear(g, i, j, k);
                if (fid == c || !adjacent(f, u)) continue;
                const unsigned n = held(start, fid);
                if (n == 0) {
                    level[c] = 1;
                    return;
                }
                if (n <= (unsigned)delta && on_border(g, f)) {
                    level[c] = 2;
                    return;
                }
            }
        }
    }
    for (int j = u[1] - 1; j <= u[1] + 1; j++)
        for (int i = u[0] - 1; i <= u[0] + 1; i++)
            for (int k = u[2] - 1; k <= u[2] + 1; k++) {
                const unsigned fid = linear(g, i, j, k);
                if (fid == c || held(start, fid) > (unsigned)delta) continue;
                for (int b = j - 1; b <= j + 1; b++) {
                    if (b < 0 || b >= g.ny) continue;
                    for (int a = i - 1; a <= i + 1; a++) {
                        if (a < 0 || a >= g.nx) continue;
                        for (int e = k - 1; e <= k + 1; e++) {
                            if (e < 0 || e >= g.nz) continue;
                            if (held(start, linear(g, a, b, e)) == 0) {
                                level[c] = 2;
                                return;
                            }
                        }
                    }
                }
            }
}

// LNMOnceKernel / LNMComputeOnce (lnm.h:332-378) at reference level L
__global__ void k_lnm_once(GridDev g, const unsigned *__restrict__ start, int *__restrict__ level, int L,
                           int *__restrict__ changed) {
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.total) return;
    if (L == 0) level[c] = -1;   // LNMInvalidateCells
    if (level[c] > -1) return;
    int u[3];
    coords(g, c, u);
    int v = -1;
    if (held(start, c) == 0) v = 0;
    else if (on_border(g, u)) v = 1;
    else if (L > 0) {
        for (int k = u[2] - 1; k <= u[2] + 1 && v < 0; k++)
            for (int j = u[1] - 1; j <= u[1] + 1 && v < 0; j++)
                for (int i = u[0] - 1; i <= u[0] + 1; i++) {
                    const unsigned nb = linear(g, i, j, k);
                    if (nb != c && level[nb] == L - 1) {
                        v = L;
                        break;
                    }
                }
    }
    if (v >= 0) {
        level[c] = v;
        *changed = 1;
    }
}

// LNMParticleAttributesKernel (lnm.h:418-432): the level of the cell of each particle's
// hashed position (positive levels only)
__global__ void k_lnm_attributes(int n, GridDev g, float iz, const float4 *__restrict__ pos,
                                 const int *__restrict__ level, int *__restrict__ val) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    unsigned bad = 0;
    const int L = level[grid_hash(g, pos[q], iz, &bad)];
    val[q] = L > 0 ? L : 0;
}

// LNMBoundaryLKKernel (lnm.h:304-330): a non-L1 cell with particles next to an L1 cell holding
// at most delta particles becomes -2 (its particles L2)
__global__ void k_lnm_lk(GridDev g, const unsigned *__restrict__ start, int *__restrict__ level, int delta) {
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.total) return;
    if (held(start, c) == 0 || level[c] == 1) return;
    int u[3];
    coords(g, c, u);
    for (int k = max(u[2] - 1, 0); k <= min(u[2] + 1, g.nz - 1); k++)
        for (int j = max(u[1] - 1, 0); j <= min(u[1] + 1, g.ny - 1); j++)
            for (int i = max(u[0] - 1, 0); i <= min(u[0] + 1, g.nx - 1); i++) {
                const unsigned nb = linear(g, i, j, k);
                if (level[nb] == 1 && held(start, nb) <= (unsigned)delta) {
                    level[c] = -2;
                    return;
                }
            }
}

// the extended variant's particle levels: L1 cells 1, filtered cells 2, unfiltered level-2
// cells 3 (LNMBoundaryExtendL2Kernel), else the attribute of the hashed position
__global__ void k_lnm_extended_out(int n, const unsigned *__restrict__ cell, const int *__restrict__ pid,
                                   const int *__restrict__ level, const int *__restrict__ val, int *__restrict__ out) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int L = level[cell[q] & ~kWide];
    out[pid[q]] = L == 1 ? 1 : L == -2 ? 2 : L == 2 ? 3 : val[q];
}

// per slot: the L1 cells' particles 1, the rest 0; the particles of L2 cells queued
__global__ void k_lnm_queue(int n, const unsigned *__restrict__ cell, const int *__restrict__ pid,
                            const int *__restrict__ level, int *__restrict__ queue, int *__restrict__ counts,
                            int *__restrict__ out) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int L = level[cell[q] & ~kWide];
    out[pid[q]] = L == 1 ? 1 : 0;
    if (L == 2) queue[atomicAdd(&counts[0], 1)] = q;
}

__device__ __forceinline__ float exact_distance(float4 a, float4 b) {
    const float ex = fs(a.x, b.x), ey = fs(a.y, b.y), ez = fs(a.z, b.z);
    return __fsqrt_rn(fa(fa(fm(ex, ex), fm(ey, ey)), fm(ez, ez)));
}

// the 27 cells around the cell of p (GetNeighborsOf order: y, then x, then z), each cell's
// slots in chain order; fn(slot) returns true to stop
template <typename Fn>
__device__ __forceinline__ void around(const BoundaryArgs &A, float4 p, Fn fn) {
    unsigned bad = 0;
    int u[3];
    coords(A.g, grid_hash(A.g, p, A.iz, &bad), u);
    for (int j = max(u[1] - 1, 0); j <= min(u[1] + 1, A.g.ny - 1); j++)
        for (int i = max(u[0] - 1, 0); i <= min(u[0] + 1, A.g.nx - 1); i++)
            for (int k = max(u[2] - 1, 0); k <= min(u[2] + 1, A.g.nz - 1); k++) {
                const unsigned nb = linear(A.g, i, j, k);
                for (unsigned s = A.start[nb]; s < A.start[nb + 1]; s++)
                    if (fn(s)) return;
            }
}

// The same walk for fn(position), the starts of a column's three cells and then four positions requested
// together: the queued test of 60,000 particles, whose few warps wait for loads, 178 -> 159 us with the
// passes around it; every particle of 262,144, bound by issue, 153 -> 149.
template <typename Fn>
__device__ __forceinline__ void around4(const BoundaryArgs &A, float4 p, Fn fn) {
    unsigned bad = 0;
    int u[3];
    coords(A.g, grid_hash(A.g, p, A.iz, &bad), u);
    const unsigned plane = (unsigned)A.g.nx * (unsigned)A.g.ny;
    const unsigned z0 = (unsigned)max(u[2] - 1, 0), z1 = (unsigned)min(u[2] + 1, A.g.nz - 1);
    for (int j = max(u[1] - 1, 0); j <= min(u[1] + 1, A.g.ny - 1); j++)
        for (int i = max(u[0] - 1, 0); i <= min(u[0] + 1, A.g.nx - 1); i++) {
            const unsigned row = (unsigned)i + (unsigned)j * (unsigned)A.g.nx;
            unsigned b[3], e[3];
#pragma unroll
            for (int z = 0; z < 3; z++) {
                const unsigned nb = row + min(z0 + z, z1) * plane;
                b[z] = __ldg(&A.start[nb]);
                e[z] = z0 + z <= z1 ? __ldg(&A.start[nb + 1]) : b[z];
            }
#pragma unroll 1
            for (int z = 0; z < 3; z++) {
                const unsigned end = z == 0 ? e[0] : z == 1 ? e[1] : e[2];
                for (unsigned s = z == 0 ? b[0] : z == 1 ? b[1] : b[2]; s < end; s += 4) {
                    float4 x[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) x[k] = __ldg(&A.pos[min(s + k, end - 1u)]);
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (s + k < end) fn(x[k]);
                }
            }
        }
}

// XiaoweiParticleIsBoundary (xiaowei.h:21-78).  Bound: FP32 issue slots (77 %) of the exact distances,
// divisions and weights of 216 candidates; 262,144 particles: 677 us with the weights' products in
// double (the FP64 pipe 86 % busy) -> 149 us.
__device__ int xiaowei(const BoundaryArgs &A, unsigned q) {
    if (A.rho[q] < A.x_rhot) return 1;
    const float4 pi = A.pos[q];
    float sx = 0.f, sy = 0.f, sz = 0.f, wsum = 0.f;
    around4(A, pi, [&](const float4 pj) {
        const float d = exact_distance(pi, pj);
        // SphStdKernel3::W at radius 6h (kernel.cpp:123-132)
        const float d2 = fm(d, d);
        const float of = fs(d2, A.x_h2);
        float w = 0.f;
        if (!(fabsf(of) < A.iz || of > 0.f)) {
            w = double_cube(A.x_wc, A.x_wh, A.x_wl, fs(1.f, fdv(d2, A.x_h2)));
        }
        sx = fa(sx, fm(pj.x, w));
        sy = fa(sy, fm(pj.y, w));
        sz = fa(sz, fm(pj.z, w));
        wsum = fa(wsum, w);
    });
    const float inv = fdv(1.f, wsum);
    const float4 m = make_float4(fm(sx, inv), fm(sy, inv), fm(sz, inv), 0.f);
    return (double)exact_distance(pi, m) > A.x_limit ? 1 : 0;
}

// DiltsSpokeParticleIsBoundary (dilts.h:110-153) by a warp: the particle is on the boundary when
// one of the 65 x 65 points of the sphere around it lies in no neighbour's sphere, whichever
// point and in whichever order, so the lanes take points side by side and stop together.  The
// overlapping neighbours (the first 1024 in walk order) are gathered by the lanes, kDiltsShared of
// them in shared memory; past that a point the stored ones leave open walks the cells again
// for the rest.  A lane tries the sphere that held its last point first.  Distances are
// compared squared with the largest float whose root does not pass the bound.
// Bound: FP32 issue slots, 89 % of them.  The angles are read from shared
// memory: from the kernel's parameters, where every lane wants another, they took 1.2 ms of 1.8.
// Measured, 32,736 particles of a BCC block: 6.3 ms (a thread per particle, points one after
// another out of a local array) -> 0.93 ms (a run of consecutive points per lane: the same).
constexpr int kDiltsShared = 96, kDiltsWarps = 4, kDiltsCap = 1024;

// Scattered particles (few candidates, the first point open) are told by a thread each: a warp for each
// took 376 us for 262,144 of them, 75 now.  A block takes `turn` particles: a thread of its first warp for
// each, its four warps for what is left; more than four when that leaves 32 blocks an SM (with 16, dense
// particles, whose tests differ in length, waited for the last blocks: 64,000 of them 2,275 us, 2,100 so).
constexpr unsigned kDiltsScattered = 16;
__host__ __device__ inline int dilts_turn(int total) {
    int turn = kDiltsWarps;
    while (turn < 32 && total > turn * 2 * 32 * kSms) turn *= 2;
    return turn;
}

__device__ __forceinline__ float exact_distance2(float4 a, float4 b) {
    const float ex = fs(a.x, b.x), ey = fs(a.y, b.y), ez = fs(a.z, b.z);
    return fa(fa(fm(ex, ex), fm(ey, ey)), fm(ez, ez));
}

__device__ __forceinline__ float4 dilts_point(const BoundaryArgs &A, float4 p, const float *spoke, int u, int v) {
    const float su = spoke[u], cu = spoke[65 + u], sv = spoke[130 + v], cv = spoke[195 + v], rad = A.d_rad;
    return make_float4(fa(fm(fm(su, cv), rad), p.x), fa(fm(fm(su, sv), rad), p.y), fa(fm(cu, rad), p.z), 0.f);
}

// True when particle q has few candidates in its 27 cells and none of them holds the first point: it is
// on the boundary.
__device__ bool dilts_scattered(const BoundaryArgs &A, unsigned q, const float *spoke) {
    const float4 pi = A.pos[q];
    unsigned bad = 0, candidates = 0;
    int u[3];
    coords(A.g, grid_hash(A.g, pi, A.iz, &bad), u);
    const int x0 = max(u[0] - 1, 0), x1 = min(u[0] + 1, A.g.nx - 1);
    unsigned b[9], e[9];   // rows of three cells
#pragma unroll
    for (int r = 0; r < 9; r++) {
        const int j = u[1] - 1 + r / 3, k = u[2] - 1 + r % 3;
        b[r] = e[r] = 0;
        if (j >= 0 && j < A.g.ny && k >= 0 && k < A.g.nz) {
            b[r] = A.start[linear(A.g, x0, j, k)];
            e[r] = A.start[linear(A.g, x1, j, k) + 1u];
        }
        candidates += e[r] - b[r];
    }
    if (candidates > kDiltsScattered) return false;
    const float4 pt = dilts_point(A, pi, spoke, 0, 0);
    bool open = true;
#pragma unroll
    for (int r = 0; r < 9; r++)
        for (unsigned s = b[r]; s < e[r]; s++) {
            const float4 pj = A.pos[s];
            if (s != q && !(exact_distance2(pi, pj) > A.d_lim2) && exact_distance2(pj, pt) <= A.d_rad2) open = false;
        }
    return open;
}

__device__ int dilts(const BoundaryArgs &A, unsigned q, const float *spoke, float4 *near) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const float4 pi = A.pos[q];
    int n = 0;   // neighbours so far
    unsigned bad = 0;
    int u[3];
    coords(A.g, grid_hash(A.g, pi, A.iz, &bad), u);
    __syncwarp();   // the warp's previous particle is done with `near`
    // a cell's slots per lane, in walk order; then the cells that hold any, one after another
    unsigned b = 0, len = 0;
    if (lane < 27) {
        const int j = u[1] - 1 + lane / 9, i = u[0] - 1 + lane / 3 % 3, k = u[2] - 1 + lane % 3;
        if (i >= 0 && i < A.g.nx && j >= 0 && j < A.g.ny && k >= 0 && k < A.g.nz) {
            const unsigned nb = linear(A.g, i, j, k);
            b = A.start[nb];
            len = A.start[nb + 1] - b;
        }
    }
    for (unsigned cells = __ballot_sync(full, len > 0); cells; cells &= cells - 1u) {
        const int from = __ffs((int)cells) - 1;
        const unsigned first = __shfl_sync(full, b, from), e = first + __shfl_sync(full, len, from);
        for (unsigned s = first; s < e && n < kDiltsCap; s += 32u) {
            const unsigned t = s + (unsigned)lane;
            float4 pj = pi;
            bool hit = t < e && t != q;
            if (hit) {
                pj = A.pos[t];
                hit = !(exact_distance2(pi, pj) > A.d_lim2);
            }
            const unsigned m = __ballot_sync(full, hit);
            const int at = n + __popc(m & ((1u << lane) - 1u));
            if (hit && at < kDiltsShared) near[at] = pj;
            n = min(n + __popc(m), kDiltsCap);
        }
    }
    __syncwarp();
    const int nl = min(n, kDiltsShared);
    int last = 0;
    for (int p0 = 0; p0 < 65 * 65; p0 += 32) {
        const int p = p0 + lane, pu = p / 65, pv = p - 65 * pu;
        bool open = false;
        if (p < 65 * 65) {
            const float4 pt = dilts_point(A, pi, spoke, pu, pv);
            open = !(nl > 0 && exact_distance2(near[last], pt) <= A.d_rad2);
            if (open)
                for (int t = 0; t < nl; t++)
                    if (exact_distance2(near[t], pt) <= A.d_rad2) {
                        open = false;
                        last = t;
                        break;
                    }
            if (open && n > kDiltsShared) {
                int seen = 0;
                around(A, pi, [&](unsigned s) {
                    if (s == q) return false;
                    const float4 pj = A.pos[s];
                    if (exact_distance2(pi, pj) > A.d_lim2) return false;
                    if (seen++ < kDiltsShared) return false;
                    if (exact_distance2(pj, pt) <= A.d_rad2) open = false;
                    return !open || seen >= kDiltsCap;
                });
            }
        }
        if (__any_sync(full, open)) return 1;
    }
    return 0;
}

// LNMBoundaryL2GeomKernel (lnm.h:57-79): each queued particle marked 2 when the test says so
__global__ void k_lnm_xiaowei(BoundaryArgs A, const int *__restrict__ queue, int *__restrict__ counts,
                              int *__restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= counts[0]) return;
    const unsigned q = (unsigned)queue[t];
    if (xiaowei(A, q) > 0) {
        out[A.pid[q]] = 2;
        atomicAdd(&counts[1], 1);
    }
}

// XiaoweiBoundary / DiltsSpokeBoundary over every particle
__global__ void k_xiaowei(BoundaryArgs A, int n, int *__restrict__ out) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    out[A.pid[q]] = xiaowei(A, (unsigned)q);
}

// Dilts over every particle, or with `queue` (of counts[0] particles) as k_lnm_xiaowei.  32 registers, for
// 16 blocks an SM: the lanes' walk of the spheres wants the warps (262,144 particles 1,050 us at 40, 975).
__global__ void __launch_bounds__(32 * kDiltsWarps, 16)
k_dilts(BoundaryArgs A, int n, const int *__restrict__ queue, int *__restrict__ counts, int *__restrict__ out) {
    __shared__ float4 near[kDiltsWarps][kDiltsShared];
    __shared__ float spoke[260];
    __shared__ unsigned todo[32];
    __shared__ int left;
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, total = queue ? counts[0] : n;
    const int turn = dilts_turn(total);
    auto tell = [&](unsigned q, bool on) {
        if (!queue) {
            out[A.pid[q]] = on ? 1 : 0;
        } else if (on) {
            out[A.pid[q]] = 2;
            atomicAdd(&counts[1], 1);
        }
    };
    if ((long long)blockIdx.x * turn >= total) return;
    for (int k = threadIdx.x; k < 260; k += blockDim.x) spoke[k] = A.spoke[k];
    __syncthreads();
    for (long long t0 = (long long)blockIdx.x * turn; t0 < total; t0 += (long long)gridDim.x * turn) {
        if (wid == 0) {
            const bool mine = lane < turn && t0 + lane < total;
            unsigned q = 0;
            bool done = true;
            if (mine) {
                q = queue ? (unsigned)queue[t0 + lane] : (unsigned)(t0 + lane);
                done = dilts_scattered(A, q, spoke);
                if (done) tell(q, true);
            }
            const unsigned rest = __ballot_sync(0xffffffffu, !done);
            if (!done) todo[__popc(rest & ((1u << lane) - 1u))] = q;
            if (lane == 0) left = __popc(rest);
        }
        __syncthreads();
        for (int k = wid; k < left; k += kDiltsWarps) {
            const int b = dilts(A, todo[k], spoke, near[wid]);
            if (lane == 0) tell(todo[k], b > 0);
        }
        __syncthreads();   // todo and left are read
    }
}

}  // namespace

void launch_lnm_single(const GridDev &g, const unsigned *start, const unsigned *cell, const int *pid, int n,
                       int delta, int *level, int *out, cudaStream_t s) {
    k_lnm_single<<<blocks_for(g.total, 256), 256, 0, s>>>(g, start, level, delta);
    k_lnm_particles<<<blocks_for(n, 256), 256, 0, s>>>(n, cell, pid, level, out);
}

void launch_lnm_once(const GridDev &g, const unsigned *start, int *level, int L, int *changed, cudaStream_t s) {
    k_lnm_once<<<blocks_for(g.total, 256), 256, 0, s>>>(g, start, level, L, changed);
}

void launch_lnm_extended_finish(const GridDev &g, float iz, const float4 *pos, const unsigned *start,
                                const unsigned *cell, const int *pid, int n, int delta, int *level, int *val,
                                int *out, cudaStream_t s) {
    k_lnm_attributes<<<blocks_for(n, 256), 256, 0, s>>>(n, g, iz, pos, level, val);
    k_lnm_lk<<<blocks_for(g.total, 256), 256, 0, s>>>(g, start, level, delta);
    k_lnm_extended_out<<<blocks_for(n, 256), 256, 0, s>>>(n, cell, pid, level, val, out);
}

void launch_lnm_geometric(const BoundaryArgs &A, const unsigned *cell, int n, int delta, int algorithm,
                          int *level, int *queue, int *counts, int *out, cudaStream_t s) {
    k_lnm_l1<<<blocks_for(A.g.total, 256), 256, 0, s>>>(A.g, A.start, level);
    k_lnm_l2<<<blocks_for(A.g.total, 256), 256, 0, s>>>(A.g, A.start, level, delta);
    cudaMemsetAsync(counts, 0, 2 * sizeof(int), s);
    k_lnm_queue<<<blocks_for(n, 256), 256, 0, s>>>(n, cell, A.pid, level, queue, counts, out);
    // the queue's length is on the device: enough warps for all of it, at most 16 blocks an SM
    if (algorithm == 1) k_lnm_xiaowei<<<blocks_for(n, 128), 128, 0, s>>>(A, queue, counts, out);
    else k_dilts<<<std::min(blocks_for(n, kDiltsWarps), 16 * kSms), 32 * kDiltsWarps, 0, s>>>(A, n, queue, counts, out);
}

void launch_boundary_test(const BoundaryArgs &A, int algorithm, int n, int *out, cudaStream_t s) {
    if (algorithm == 1) k_xiaowei<<<blocks_for(n, 128), 128, 0, s>>>(A, n, out);
    else k_dilts<<<blocks_for(n, dilts_turn(n)), 32 * kDiltsWarps, 0, s>>>(A, n, nullptr, nullptr, out);
}

void launch_lnm(const GridDev &g, const unsigned *start, const unsigned *cell, const int *pid, int n, int delta,
                int *level, int *out, cudaStream_t s) {
    k_lnm_l1<<<blocks_for(g.total, 256), 256, 0, s>>>(g, start, level);
    k_lnm_l2<<<blocks_for(g.total, 256), 256, 0, s>>>(g, start, level, delta);
    k_lnm_particles<<<blocks_for(n, 256), 256, 0, s>>>(n, cell, pid, level, out);
}

}  // namespace bbg
