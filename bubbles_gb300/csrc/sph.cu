// sph.cu -- neighbour-sum passes of the 3D SPH / PCISPH step (FP32, one thread per
// particle over the cell-sorted arrays; several lanes per particle for the fewest, kGroup16).
//
// Neighbour sets follow the reference buckets: j is a neighbour of i when
// IsWithinStd(|x_i - x_j|, h) holds at the positions of the last grid update
// (src/core/grid.h:423-447).  The density pass filters the candidates of the 27 cells (9
// contiguous slot ranges) once per substep, applies the exact FP32 membership test to what
// is left and records the members in a compact list (tile.cuh); later passes walk that list.  The
// predicted-density pass uses the step-start membership with values at predicted
// positions, which is what the reference does with its stale bucket
// (src/equations/pcisph_equations3.cpp:58-89).
//
// Fusions (per PCISPH substep: density, non-pressure, 2 per corrector iteration):
//   - non-pressure force + the k = 0 prediction (PredictVelocityAndPositionFor);
//   - pressure force of iteration k + either the prediction of iteration k+1 or, once
//     the density error of iteration k is below tolerance (or k is the last allowed
//     iteration), AccumulateForcesFor + TimeIntegrationFor into the other buffer.
// The iteration decision is read from device memory (max error of each iteration), so
// the host launches max_iterations x 2 kernels without synchronising; kernels of
// iterations after convergence return immediately.
#include <climits>

#include "bbg_kernels.h"
#include "tile.cuh"

namespace bbg {

constexpr int kThreads = kTile;

#ifndef BBG_NBR_MIN_BLOCKS
#define BBG_NBR_MIN_BLOCKS 8
#endif
#ifndef BBG_PF_MIN_BLOCKS
#define BBG_PF_MIN_BLOCKS 12
#endif
// resident 128-thread blocks per SM the member-walking passes are compiled for (register
// budget; build-time tuning knobs, measured: 12 for the pressure-force pass, which trades
// a few spilled registers for occupancy, 8 for the others).  Kernels are compiled for
// blocks of up to kMaxTile threads with the same register budget.
constexpr int kNbrMinBlocks = BBG_NBR_MIN_BLOCKS * kTile / kMaxTile;
#ifndef BBG_PD_MIN_BLOCKS
#define BBG_PD_MIN_BLOCKS 16
#endif
// the predicted-density pass fits 32 registers without spilling (gather batch 4): full
// occupancy for its latency-bound gathers
constexpr int kPdMinBlocks = BBG_PD_MIN_BLOCKS * kTile / kMaxTile;
constexpr int kPfMinBlocks = BBG_PF_MIN_BLOCKS * kTile / kMaxTile;
#ifndef BBG_PDWL_MIN_BLOCKS
#define BBG_PDWL_MIN_BLOCKS 16
#endif
#ifndef BBG_PFWL_MIN_BLOCKS
#define BBG_PFWL_MIN_BLOCKS 12
#endif
// register budgets of the persistent batch passes, as the per-tile passes' (measured on
// config 4: 8 blocks per SM, 48 and 64 registers without spills, lost 6 % to these, which
// spill a little)
constexpr int kPdWlMinBlocks = BBG_PDWL_MIN_BLOCKS * kTile / kMaxTile;
constexpr int kPfWlMinBlocks = BBG_PFWL_MIN_BLOCKS * kTile / kMaxTile;
#ifndef BBG_DENSITY_MIN_BLOCKS
#define BBG_DENSITY_MIN_BLOCKS 8
#endif
// density pass: at most 64 registers (it takes 56, 9 blocks an SM; capped for 12 it spills)
constexpr int kDensityMinBlocks = BBG_DENSITY_MIN_BLOCKS * kTile / kMaxTile;

// Up to this many particles the member passes are bound by the latency of each particle's dependent
// loads, with few warps an SM to hide it: kernels that request more of them together (the compiler
// takes 90 to 103 registers: five blocks of 128 an SM, four at the most).  The line is one wave of four
// blocks an SM.  A substep of 19,720 particles, 8 corrector iterations: 218 -> 193 us; 65,600: 222 -> 208; 5,814, 1
// iteration: 79 -> 71; past the line they lose (122,500: 271 -> 341).
constexpr int kFew = kSms * 4 * kTile;
constexpr int kFewBatch = 16, kFewBatchPosVel = 8;   // members together (one or two records each)

// a neighbour's position and velocity records
struct PosVel {
    float4 p, v;
};

static inline int blocks_for(long long n, int t) { return (int)((n + t - 1) / t); }

__device__ __forceinline__ bool finite_state(v3 x, v3 v) {
    return isfinite(x.x) && isfinite(x.y) && isfinite(x.z) && isfinite(v.x) && isfinite(v.y) && isfinite(v.z);
}

// warp-aggregated count of the lanes with a non-finite integrated state (all lanes call it)
__device__ __forceinline__ void count_nonfinite(bool bad, StepState *st) {
    const unsigned m = __ballot_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(&st->nonfinite, (unsigned)__popc(m));
}

// True when some corrector iteration before k already met the tolerance
// (ComputePressureForceAndIntegrate's break, pcisph_equations3.cpp:243-246).
__device__ __forceinline__ bool converged_before(const Params &P, const StepState *st, int k) {
    for (int q = 0; q < k; q++) {
        float e = __uint_as_float(st->err_bits[q]);
        if (fdv(e, P.target_density) < P.max_err_ratio) return true;
    }
    return false;
}

// Batch: true when scene s met the tolerance at an iteration before k (its particles
// are integrated and skip the rest of the corrector).
__device__ __forceinline__ bool scene_converged_before(const Params &P, int s, int k) {
    const SceneState &ss = P.scene_st[s];
    for (int q = 0; q < k; q++) {
        float e = __uint_as_float(ss.err_bits[q]);
        if (fdv(e, P.target_density) < P.max_err_ratio) return true;
    }
    return false;
}

// The member phase of the density pass for particle i: the exact membership test, the kernel
// sum (i included) and the member list of candidates in the order of the 27 cells' rows, which
// is ascending slots.  Lanes whose candidates are nearly all members write the same one or two list rows
// together.
struct DensitySum {
    float sum = 0.f;
    int listed = 0;   // members other than i
    int self = 0;     // 1 when i is its own member (not at a position that is not finite)
    ListEntry *out;
    __device__ __forceinline__ explicit DensitySum(ListEntry *o) : out(o) {}
    __device__ __forceinline__ static float dist(float4 pi, float4 pj) {
        const float dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
        return __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
    }
    __device__ __forceinline__ void take(const Params &P, bool mem, float r2, unsigned j, unsigned i) {
        const float x = __fmaf_rn(-r2, P.inv_h2, 1.f);
        const float t = __fmul_rn(__fmul_rn(x, x), x);
        sum = mem ? __fadd_rn(sum, t) : sum;
        const bool other = mem && j != i;
        if (other && listed < kMaxList) *out = j;
        out += other ? P.n : 0;
        listed += other ? 1 : 0;
        self += mem && !other ? 1 : 0;
    }
};

// The end of the density pass for particle i: density, equation of state, counters.
__device__ __forceinline__ void density_store(const Params &P, float4 *pos, float4 *vel, unsigned *cell, float *rho,
                                              float *inv_rho, float *press, int *nbr, int compute_pressure,
                                              StepState *st, int i, float4 pi, unsigned cw, float sum, int cnt,
                                              int listed) {
    const float di = sum * P.std_c * P.mass;
    if (compute_pressure) {
        float p = P.eos_scale_over_exp * (powf(di / P.target_density, P.eos_exp) - 1.f);
        if (p < 0.f) p *= P.neg_scale;
        press[i] = p;
        reinterpret_cast<float *>(&pos[i])[3] = p / (di * di);   // pos.w = p / rho^2
    }
    rho[i] = di;
    const float ir = 1.f / di;
    inv_rho[i] = ir;
    reinterpret_cast<float *>(&vel[i])[3] = ir;                   // vel.w = 1 / rho
    nbr[i] = cnt;
    if (P.nscenes > 0) P.scene[i] = (unsigned short)scene_of(P, pi.z);
    if (listed > kMaxList) cell[i] = cw | kWide;
    if (cnt > kBucketCap) atomicAdd(&st->nbr_overflow, 1u);
}

// The member phase over `kept` non-empty masks of candidates, entry k at keep[k * stride]: (mask,
// slot of bit 31, the next slots below it).  NB records requested together.
template <int NB>
__device__ __forceinline__ void density_members(const Params &P, const float4 *__restrict__ pos, float4 pi, unsigned i,
                                                DensitySum &D, const uint2 *keep, int stride, int kept) {
    const uint2 *const end = keep + kept * stride;
    unsigned m = 0, base = 0;
    while (m != 0 || keep != end) {
        unsigned j[NB];
        bool mem[NB];
#pragma unroll
        for (int u = 0; u < NB; u++) {
            if (m == 0 && keep != end) {
                const uint2 v = *keep;
                m = v.x;
                base = v.y;
                keep += stride;
            }
            mem[u] = m != 0;
            const unsigned c = (unsigned)__clz((int)m) & 31u;
            j[u] = mem[u] ? base + c : i;
            m &= ~(0x80000000u >> c);
        }
        float4 p[NB];
#pragma unroll
        for (int u = 0; u < NB; u++) p[u] = __ldg(&pos[j[u]]);
        float r2[NB];
        bool all = true;   // members without the exact test
#pragma unroll
        for (int u = 0; u < NB; u++) {
            r2[u] = DensitySum::dist(pi, p[u]);
            all = all && r2[u] < P.nb_lo;
        }
        if (!all) {
#pragma unroll
            for (int u = 0; u < NB; u++) mem[u] = mem[u] && std_member(P, pi, p[u], r2[u]);
        }
#pragma unroll
        for (int u = 0; u < NB; u++) D.take(P, mem[u], r2[u], j[u], i);
    }
}

// The filter's records of positions that the last grid update did not write them for.
__global__ void __launch_bounds__(kThreads)
k_filter_records(Params P, const float4 *__restrict__ pos, const unsigned *__restrict__ cell, __half *__restrict__ rec) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < P.n) filter_record(P, pos[i], cell[i] & ~kWide, (unsigned)i, rec);
}

__device__ __forceinline__ unsigned half2_bits(__half2 v) { return *reinterpret_cast<unsigned *>(&v); }
__device__ __forceinline__ __half2 as_half2(unsigned v) { return *reinterpret_cast<__half2 *>(&v); }

// Masks a particle keeps between the filter and the member phase of k_density_mask: 9 rows and
// one more for a row whose slots span more than 32.  Denser particles (the rest density compressed by a
// third, or a wider kernel) take the two phases in several rounds: 1,000,000 particles at 1.63 times the rest
// density 265 us (walked one candidate after another they took 628), at 1.17 times, one round, 158.
// The further rounds are compiled to fit the first one's 56 registers, 9 blocks an SM: with 61 to 64 of them
// the single-round states took 3 % longer.
constexpr int kMasks = 10;

// The filter of k_density_mask for the particle at pi in cell c: the non-empty masks of its
// candidates, entry k at keep[k * stride].  Returns their number, or when kMasks have no room for
// them ~s, s the slot to go on from: with RESUME, from there, one mask fewer at a time.
// total: the candidates of the 27 cells.
template <bool FEW, bool RESUME>
__device__ __forceinline__ int density_filter(const Params &P, const unsigned *__restrict__ start,
                                              const uint4 *__restrict__ rec, float4 pi, unsigned c, uint2 *keep,
                                              int stride, unsigned from, unsigned &total) {
    constexpr int room = RESUME ? kMasks - 1 : kMasks;
    int kept = 0;
    total = 0;
    const GridDev &g = P.g;
    int cx, cy, cz;
    cell_coords(g, c, cx, cy, cz);
    const v3 f = filter_offset(P, pi, cx, cy, cz);
    const int far = ((cx + 1) & 2) ? 0 : 1;   // cells 1 and 2 of the first window, else the second
    const __half2 X = __float2half2_rn((float)(((cx + 2 * far) & 3) - 2) * P.filt_side[0] + f.x);
    const __half2 T = as_half2(P.filt);
    // rows x, y, z of a record, or y, z, x' of the second window: the test takes the axes in any order
    const uint4 *const rec0 = rec + far;
    const int x0 = cx > 0 ? -1 : 0, x1 = cx + 1 < g.nx ? 2 : 1;
    const int plane = g.nx * g.ny;
    // row r = 3 (dz + 1) + dy + 1, inside the grid or empty; the next row's range is requested a row
    // ahead (with RESUME not, for its registers)
    unsigned inside = 0x1ffu;
    if (cy == 0) inside &= ~0x049u;
    if (cy + 1 >= g.ny) inside &= ~0x124u;
    if (cz == 0) inside &= ~0x007u;
    if (cz + 1 >= g.nz) inside &= ~0x1c0u;
    int row = (int)c - g.nx - plane;
    unsigned nb = 0, ne = 0;
    auto range = [&]() {
        nb = ne = 0;
        if (inside & 1u) {
            nb = __ldg(&start[row + x0]);
            ne = __ldg(&start[row + x1]);
        }
    };
    if (!RESUME) range();
    __half2 Z = __float2half2_rn(f.z + 0.5f * P.filt_side[2]);
    float fy = f.y + 0.5f * P.filt_side[1];
    int dy = 0;
#pragma unroll 1
    for (int r = 0; r < 9; r++) {
        if (RESUME) range();
        const unsigned b = nb, e = ne;
        const __half2 Y = __float2half2_rn(fy);
        const __half2 A = far ? Y : X, B = far ? Z : Y, C = far ? X : Z;
        fy -= P.filt_side[1];
        row += g.nx;
        if (++dy == 3) {
            dy = 0;
            row += plane - 3 * g.nx;
            fy = f.y + 0.5f * P.filt_side[1];
            Z = __float2half2_rn(f.z + (r == 2 ? -0.5f : -1.5f) * P.filt_side[2]);
        }
        inside >>= 1;
        if (!RESUME) range();
        total += e - b;
        for (unsigned cb = RESUME && from > b ? from : b & ~7u; cb < e; cb += 32u) {
            const unsigned span = min(32u, e - cb);
            const int groups = (int)((span + 7u) >> 3);
            const uint4 *q = rec0 + (size_t)(cb >> 3) * 4u;
            unsigned m = 0;
            auto group = [&](const uint4 &a, const uint4 &v, const uint4 &w) {
                auto test = [&](unsigned ua, unsigned ub, unsigned uc) {
                    const __half2 da = __hsub2(as_half2(ua), A), db = __hsub2(as_half2(ub), B);
                    const __half2 dc = __hsub2(as_half2(uc), C);
                    return half2_bits(__hfma2(__hneg2(da), da, __hfma2(__hneg2(db), db, __hfma2(__hneg2(dc), dc, T))));
                };
                const unsigned w0 = test(a.x, v.x, w.x), w1 = test(a.y, v.y, w.y);
                const unsigned w2 = test(a.z, v.z, w.z), w3 = test(a.w, v.w, w.w);
                // the eight signs (set: outside) as a byte, the first slot its top bit
                unsigned s = __dp4a(__byte_perm(w0, w1, 0x7531) & 0x80808080u, 0x10204080u, 0u);
                s = __dp4a(__byte_perm(w2, w3, 0x7531) & 0x80808080u, 0x01020408u, s);
                m = (m << 8) + (s >> 7);
            };
            if (FEW) {
                uint4 a[4], v[4], w[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint4 *g4 = q + 4 * min(k, groups - 1);
                    a[k] = __ldg(g4);
                    v[k] = __ldg(g4 + 1);
                    w[k] = __ldg(g4 + 2);
                }
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (k < groups) group(a[k], v[k], w[k]);
            } else {
                for (int k = 0; k < groups; k++, q += 4) group(__ldg(q), __ldg(q + 1), __ldg(q + 2));
            }
            m = ~m << (32 - 8 * groups);
            // the slots of [b, e) only
            if (b > cb) m &= 0xffffffffu >> (b - cb);
            m &= (unsigned)((int)0x80000000 >> (span - 1u));
            if (m) {
                if ((unsigned)kept < (unsigned)room) keep[kept++ * stride] = make_uint2(m, cb);
                else if (kept == room) kept = ~(int)max(cb, b);
            }
        }
    }
    return kept;
}

// The density pass: ComputeDensityFor + ComputePressureValue (sph_equations3.cpp:7-58), and each
// particle's neighbour set (the reference bucket, grid.h:423-447) as a member list.  A thread per
// particle, in two phases.
//
// Filter: all candidates of the 27 cells (about 216), eight at a time from the halves the grid update's gather wrote:
// the sign of P.filt - r^2, the squared radius widened by the rounding of the halves, into a
// mask of 32 aligned slots, and nothing else.  It only leaves out what cannot be a member.
// Members: the exact test, the kernel sum in float and the list over the about 29 candidates left.
//
// Measured at 1,048,576 particles: 234 -> 149 us; 4,194,304: 866 -> 554; 262,144: 78 -> 47 (with a
// records' launch of its own: 156, 578, 52).  The pass that tested and summed every candidate in float was bound by issue
// slots (256 M warp instructions, 83 %); this one issues 143 M, 77 % of the slots, with L1 at 72 % and the
// ALU at 52 % (masks and lists).  Float candidates in the filter were bound by L1, whose 128 bytes
// a clock return 12 bytes a candidate to every lane (181 us), half of that as halves.  A warp per
// cell that holds candidates in registers and ballots each particle's tests was slower (225 us): the
// setup per cell, 5.5 cells a warp, costs more than the loads it saves.
//
// FEW (fewer particles than fill the SMs): a row's records are all requested before any is used, and
// more members together, since no other warp hides their latency.
template <bool FEW>
__global__ void __launch_bounds__(kMaxTile, FEW ? 1 : kDensityMinBlocks)
k_density_mask(Params P, float4 *__restrict__ pos, float4 *__restrict__ vel, unsigned *__restrict__ cell,
               const unsigned *__restrict__ start, const uint4 *__restrict__ rec, float *__restrict__ rho,
               float *__restrict__ inv_rho, float *__restrict__ press, int *__restrict__ nbr,
               ListEntry *__restrict__ list, int compute_pressure, StepState *st) {
    extern __shared__ uint2 mask_smem[];   // [kMasks][blockDim.x]: mask, slot of its bit 31
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    uint2 *const keep = mask_smem + threadIdx.x;
    const int stride = (int)blockDim.x;
    const float4 pi = pos[i];
    const unsigned cw = cell[i], c = cw & ~kWide;
    unsigned total;
    int kept = density_filter<FEW, false>(P, start, rec, pi, c, keep, stride, 0u, total);
    DensitySum D(list + i);
    if (total > kMaxCandidates) {
        atomicAdd(&st->crowded, 1u);   // the particle itself only
        D.sum = 1.f;
        D.self = 1;
    } else {
        density_members<FEW ? 8 : 4>(P, pos, pi, (unsigned)i, D, keep, stride, kept < 0 ? kMasks : kept);
        while (kept < 0) {   // the rest; the last entry keeps the sums meanwhile
            keep[(kMasks - 1) * stride] = make_uint2(__float_as_uint(D.sum), 2u * (unsigned)D.listed + (unsigned)D.self);
            kept = density_filter<FEW, true>(P, start, rec, pi, c, keep, stride, ~(unsigned)kept, total);
            const uint2 d = keep[(kMasks - 1) * stride];
            D.sum = __uint_as_float(d.x);
            D.listed = (int)(d.y >> 1);
            D.self = (int)(d.y & 1u);
            D.out = list + i + (size_t)D.listed * P.n;
            density_members<FEW ? 8 : 4>(P, pos, pi, (unsigned)i, D, keep, stride, kept < 0 ? kMasks - 1 : kept);
        }
    }
    density_store(P, pos, vel, cell, rho, inv_rho, press, nbr, compute_pressure, st, i, pi, cw, D.sum,
                  D.listed + D.self, D.listed);
}

// The fewest particles: G lanes for each instead of a thread, which is one long chain of dependent loads,
// about 216 candidates deep, on an idle chip.  The density pass takes sixteen lanes or eight,
// the force pass, whose 29 members are the shorter chain, eight or four: as many as keep the density pass
// within one wave of 8 blocks of 128 an SM; past it the extra instructions of splitting a
// particle cost more than the latency they hide (12,144 particles: 16 and 8 lanes 375 us for seven
// SPH substeps, 8 and 4 lanes 340, a thread each 371; 16,384: 8 and 4 lanes 370, a thread each 375; 20,000:
// no difference; 35,937, 4 lanes: 461 against 374).
constexpr int kGroupThreads = 128;
constexpr int kGroupMembers = kMaxList;   // of a particle (itself counted) in shared memory at a time
constexpr int kGroup16 = kSms * 8 * kGroupThreads / 16;   // particles, up to
constexpr int kGroup8 = 2 * kGroup16;

// The density pass, G lanes per particle: the lanes take every G-th candidate of the particle's nine rows,
// all tested in float, and put the members' kernel values in shared memory in row order, where one
// lane adds them in that order: the sum of k_density_mask to the bit.  The block's particles
// are finished by the lanes of one warp and their lists written a row at a time by the others.
// Bound by latency: two to four rounds of loads, then the chain of additions.  1,287 particles: 16.3 -> 10.2 us
// (a timing event on either side included); with the force pass's lanes a substep 33.6 -> 24.3 us, of
// 16,384 particles 36.1 -> 33.9.
template <int G>
__global__ void __launch_bounds__(kGroupThreads, 8)
k_density_group(Params P, float4 *__restrict__ pos, float4 *__restrict__ vel, unsigned *__restrict__ cell,
                const unsigned *__restrict__ start, float *__restrict__ rho, float *__restrict__ inv_rho,
                float *__restrict__ press, int *__restrict__ nbr, ListEntry *__restrict__ list,
                int compute_pressure, StepState *st) {
    constexpr int S = kGroupThreads / G;           // particles of a block
    __shared__ unsigned row_end[9][S];   // candidates up to the end of the row
    __shared__ unsigned row_off[9][S];   // slot of a candidate of the row less its number
    __shared__ float term[kGroupMembers][S];
    __shared__ ListEntry member[kGroupMembers][S];
    __shared__ int found[S], itself[S];   // members (-1: past the work cap); the particle itself one
    constexpr unsigned full = 0xffffffffu, group = (1u << G) - 1u;
    const int grp = threadIdx.x / G, lane = threadIdx.x & (G - 1);
    const int shift = threadIdx.x & 31 & ~(G - 1);
    const int i0 = blockIdx.x * S;
    const bool live = i0 + grp < P.n;
    const int i = live ? i0 + grp : P.n - 1;
    const float4 pi = pos[i];
    const unsigned cw = cell[i], c = cw & ~kWide;
    const GridDev &g = P.g;
    int cx, cy, cz;
    cell_coords(g, c, cx, cy, cz);
    // rows r = 3 (dz + 1) + dy + 1, G at a time
    constexpr int R = (9 + G - 1) / G;
    unsigned b[R], len[R], total = 0;
#pragma unroll
    for (int u = 0; u < R; u++) {
        const int r = lane + G * u, dz = r / 3 - 1, dy = r - 3 * (r / 3) - 1;
        b[u] = len[u] = 0;
        if (live && r < 9 && cy + dy >= 0 && cy + dy < g.ny && cz + dz >= 0 && cz + dz < g.nz) {
            const unsigned row = c + (unsigned)(dy * g.nx) + (unsigned)(dz * g.nx * g.ny);
            b[u] = __ldg(&start[row - (cx > 0 ? 1u : 0u)]);
            len[u] = __ldg(&start[row + (cx + 1 < g.nx ? 2u : 1u)]) - b[u];
        }
    }
#pragma unroll
    for (int u = 0; u < R; u++) {
        unsigned end = len[u];
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const unsigned y = __shfl_up_sync(full, end, o, G);
            if (lane >= o) end += y;
        }
        end += total;
        if (lane + G * u < 9) {
            row_end[lane + G * u][grp] = end;
            row_off[lane + G * u][grp] = b[u] - (end - len[u]);
        }
        total = __shfl_sync(full, end, G - 1, G);
    }
    __syncwarp();
    const int self = std_member(P, pi, pi, DensitySum::dist(pi, pi)) ? 1 : 0;
    // (the loops run as long as the warp's longest group, with every lane in them)
    const unsigned work = total <= kMaxCandidates ? total : 0u, longest = __reduce_max_sync(full, work);
    int cnt = 0, r = 0;
    unsigned rend = row_end[0][grp], roff = row_off[0][grp];
    constexpr int NB = 8;
    for (unsigned k0 = 0; k0 < longest; k0 += NB * G) {
        unsigned j[NB];
        bool mem[NB];
        float4 p[NB];
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const unsigned k = k0 + u * G + lane;
            mem[u] = k < work;
            while (mem[u] && k >= rend) {
                r++;
                rend = row_end[r][grp];
                roff = row_off[r][grp];
            }
            j[u] = mem[u] ? roff + k : (unsigned)i;
            p[u] = __ldg(&pos[j[u]]);
        }
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const float r2 = DensitySum::dist(pi, p[u]);
            mem[u] = mem[u] && std_member(P, pi, p[u], r2);
            const unsigned m = (__ballot_sync(full, mem[u]) >> shift) & group;
            const int q = cnt + __popc(m & ((1u << lane) - 1u));   // members before this one
            cnt += __popc(m);
            if (mem[u] && q < kGroupMembers) {
                const float x = __fmaf_rn(-r2, P.inv_h2, 1.f);
                term[q][grp] = __fmul_rn(__fmul_rn(x, x), x);
                // the list leaves the particle itself out (and its last entry, if members are left, to come)
                if (j[u] != (unsigned)i) member[q - (j[u] > (unsigned)i ? self : 0)][grp] = j[u];
            }
        }
    }
    if (lane == 0) {
        found[grp] = !live ? 0 : total > kMaxCandidates ? -1 : cnt;
        itself[grp] = self;
    }
    const bool more = __syncthreads_or(cnt > kGroupMembers);
    const int mine = threadIdx.x & (S - 1);
    const int all = found[mine], listed = all - itself[mine];
    float sum = 0.f;
    if (threadIdx.x >= 32) {   // the lists, rows of the block's particles together
        for (int q = (threadIdx.x - 32) / S; q < min(listed, kMaxList); q += (kGroupThreads - 32) / S)
            list[(size_t)q * P.n + i0 + mine] = member[q][mine];
    } else if (threadIdx.x < S) {
        const int some = min(all, kGroupMembers);
#pragma unroll 8
        for (int q = 0; q < some; q++) sum = __fadd_rn(sum, term[q][mine]);
    }
    // The block's particles with more members than that (a dense state, a wider kernel): the candidates
    // again for the next ones.  15,625 particles of 93 members: 151 us when a lane of each walked them
    // alone, 54 now; none of a state of 28 members pays for it (14.4 us).
    if (more) {
        for (int base = kGroupMembers;; base += kGroupMembers) {
            __syncthreads();   // the terms are added, the lists written
            cnt = r = 0;
            rend = row_end[0][grp];
            roff = row_off[0][grp];
#pragma unroll 4
            for (unsigned k = lane; k < longest + lane; k += G) {
                bool mem = k < work;
                while (mem && k >= rend) {
                    r++;
                    rend = row_end[r][grp];
                    roff = row_off[r][grp];
                }
                const unsigned j = mem ? roff + k : (unsigned)i;
                const float4 pj = __ldg(&pos[j]);
                const float r2 = DensitySum::dist(pi, pj);
                mem = mem && std_member(P, pi, pj, r2);
                const unsigned m = (__ballot_sync(full, mem) >> shift) & group;
                const int q = cnt + __popc(m & ((1u << lane) - 1u)) - base;
                cnt += __popc(m);
                if (mem && q >= 0 && q < kGroupMembers) {
                    const float x = __fmaf_rn(-r2, P.inv_h2, 1.f);
                    term[q][grp] = __fmul_rn(__fmul_rn(x, x), x);
                    // the last entry of the list, where the particle itself came before
                    if (base + q == kMaxList && self && j > (unsigned)i) list[(size_t)(kMaxList - 1) * P.n + i] = j;
                }
            }
            const bool again = __syncthreads_or(cnt > base + kGroupMembers);
            if (threadIdx.x < S) {
                const int some = min(all - base, kGroupMembers);
                for (int q = 0; q < some; q++) sum = __fadd_rn(sum, term[q][mine]);
            }
            if (!again) break;
        }
    }
    if (threadIdx.x < S && i0 + mine < P.n) {
        const float4 pm = pos[i0 + mine];
        const unsigned cm = cell[i0 + mine];
        const bool crowded = all < 0;   // past the work cap: the particle itself only
        if (crowded) atomicAdd(&st->crowded, 1u);
        density_store(P, pos, vel, cell, rho, inv_rho, press, nbr, compute_pressure, st, i0 + mine, pm, cm,
                      crowded ? 1.f : sum, crowded ? 1 : all, crowded ? 0 : listed);
    }
}

// ComputeNonPressureForceFor (sph_equations3.cpp:80-110), optionally followed by the
// k = 0 PredictVelocityAndPositionFor (pcisph_equations3.cpp:3-28).
//   predict 0: forces only; 1: the reference's k = 0 prediction (p = 0, Fp = 0, x* from F);
//   WARM: the corrector's warm start has set p and pos.w = p / rho^2 for every particle,
//   so the same member walk also sums the pressure force of that start
//   (PredictPressureForceFor, pcisph_equations3.cpp:114-155) and x* comes from F + Fp.
// With DIV it also accumulates sum_j (1/rho_j) (1 - d/h)^2 / d (v_j - v_i).(x_j - x_i),
// the velocity divergence up to m * 45 / (pi h^4), a feature of the learned warm start.
template <bool DIV, bool WARM, int NB, int MINB = kNbrMinBlocks>
__global__ void __launch_bounds__(kMaxTile, MINB)
k_non_pressure(Params P, const float4 *__restrict__ pos, const float4 *__restrict__ vel,
               const unsigned *__restrict__ cell,
               const unsigned *__restrict__ start, const ListEntry *__restrict__ list, const int *__restrict__ nbr,
               float4 *__restrict__ force, float4 *__restrict__ xstar, float4 *__restrict__ pforce,
               float *__restrict__ press, float *__restrict__ divsum, int predict, float dt, float dt_over_m) {
    const int s0 = tile_of_block(P, blockIdx.x, (P.n + (int)blockDim.x - 1) / (int)blockDim.x) * blockDim.x;
    if (s0 >= P.n) return;
    const int i = s0 + threadIdx.x;
    if (i >= P.n) return;
    const float4 pi = pos[i];
    const float4 vi = vel[i];
    const float ai = pi.w;   // WARM: p_i / rho_i^2
    float fx = P.mass * P.gx - P.drag * vi.x;
    float fy = P.mass * P.gy - P.drag * vi.y;
    float fz = P.mass * P.gz - P.drag * vi.z;
    float tx = 0.f, ty = 0.f, tz = 0.f;
    float dv = 0.f;
    const float kv = P.visc_m2 * P.spiky_d2w_c;
    const float kg = P.m2 * P.spiky_dw_c;
    tile_members<NB>(
        P, start, list, nbr, pos, cell[i], i,
        [&](unsigned j) { return PosVel{__ldg(&pos[j]), __ldg(&vel[j])}; },
        [&](const PosVel &nb) {
            const float4 pj = nb.p, vj = nb.v;   // vj.w = 1 / rho_j
            const float r2 = dist2(pi, pj);
            const float inv_d = rsqrtf(r2);
            const float d = r2 > 0.f ? r2 * inv_d : 0.f;   // coincident particles: distance 0
            const float x = 1.f - d * P.inv_h;
            const float w = kv * x * vj.w;
            fx += (vj.x - vi.x) * w;
            fy += (vj.y - vi.y) * w;
            fz += (vj.z - vi.z) * w;
            if (WARM) {
                // as k_pressure_force: IsWithinSpiky(d, h) and d > 0 && !IsZero(d)
                if (d - P.h <= -P.iz && d >= P.iz) {
                    const float c = kg * (ai + pj.w) * x * x * inv_d;
                    tx += (pj.x - pi.x) * c;
                    ty += (pj.y - pi.y) * c;
                    tz += (pj.z - pi.z) * c;
                }
            }
            if (DIV && r2 > 0.f) {
                const float dot = (vj.x - vi.x) * (pj.x - pi.x) + (vj.y - vi.y) * (pj.y - pi.y) +
                                  (vj.z - vi.z) * (pj.z - pi.z);
                dv += vj.w * x * x * inv_d * dot;
            }
        });
    force[i] = make_float4(fx, fy, fz, 0.f);
    if (DIV) divsum[i] = dv;
    if (WARM) {
        const v3 fp = V(-tx, -ty, -tz);
        pforce[i] = F4(fp);
        v3 xs;
        predict_particle(P, dt, dt_over_m, V(fx, fy, fz), fp, V(pi), V(vi), &xs);
        xstar[i] = F4(xs);
    } else if (predict) {
        press[i] = 0.f;
        pforce[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        v3 xs;
        predict_particle(P, dt, dt_over_m, V(fx, fy, fz), V(0.f, 0.f, 0.f), V(pi), V(vi), &xs);
        xstar[i] = F4(xs);
    }
}

// PredictVelocityAndPositionFor (pcisph_equations3.cpp:3-28) on the forces already in
// `force`; with is_first: p = 0, Fp = 0, rho* = rho, so x* comes from F alone.
__global__ void __launch_bounds__(kThreads)
k_predict_first(Params P, const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                const float4 *__restrict__ force, float4 *__restrict__ xstar,
                float4 *__restrict__ pforce, float *__restrict__ press,
                float *__restrict__ rhostar, const float *__restrict__ rho, float *__restrict__ derr,
                int is_first, float dt, float dt_over_m) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    if (is_first) {
        rhostar[i] = rho[i];
        pforce[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        derr[i] = 0.f;
        press[i] = 0.f;
    }
    v3 xs;
    predict_particle(P, dt, dt_over_m, V(force[i]), V(pforce[i]), V(pos[i]), V(vel[i]), &xs);
    xstar[i] = F4(xs);
}

// Warm start of the corrector: p = scale * the start estimate (the previous substep's
// pressure), rho* = rho, and pos.w = p / rho^2 for the pressure-force pass that predicts
// x* from F + Fp(p).
__global__ void k_warm_start(int n, float4 *pos, const float *__restrict__ rho,
                             const float *__restrict__ pinit, float *__restrict__ press,
                             float *__restrict__ rhostar, float *__restrict__ derr, float scale) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float d = rho[i];
    const float p = scale * pinit[i];
    press[i] = p;
    rhostar[i] = d;
    derr[i] = 0.f;
    reinterpret_cast<float *>(&pos[i])[3] = p / (d * d);
}

// pos.w = p / rho*^2 from the pressure and predicted-density fields (used when those
// fields were set from outside rather than by the predicted-density pass).
__global__ void k_pack_acoef(int n, float4 *pos, const float *__restrict__ press,
                             const float *__restrict__ rhostar) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float d = rhostar[i];
    reinterpret_cast<float *>(&pos[i])[3] = press[i] / (d * d);
}

// The end of PredictPressureFor (pcisph_equations3.cpp:60-90) for particle i, from the kernel sum at
// predicted positions: density, its error, pressure and p / rho*^2.  Returns |err|.
__device__ __forceinline__ float pred_density_end(const Params &P, float4 *pos, float *__restrict__ press,
                                                  float *__restrict__ rhostar, float *__restrict__ derr, float delta,
                                                  int clamp_total, int i, float sum) {
    const float density = sum * P.std_c * P.mass;
    float err = density - P.target_density;
    float pr = delta * err;
    float p;
    if (clamp_total) {
        // warm-started corrector: the increment may be negative, the total is scaled
        // like a negative pressure, so an overestimated start can be corrected
        if (err < 0.f) err *= P.neg_scale;
        p = press[i] + pr;
        if (p < 0.f) p *= P.neg_scale;
    } else {
        if (pr < 0.f) {
            pr *= P.neg_scale;
            err *= P.neg_scale;
        }
        p = press[i] + pr;
    }
    press[i] = p;
    rhostar[i] = density;
    derr[i] = err;
    reinterpret_cast<float *>(&pos[i])[3] = p / (density * density);   // pos.w = p / rho*^2
    return fabsf(err);
}

// PredictPressureFor (pcisph_equations3.cpp:60-90) of particle i over the step-start
// neighbour set at predicted positions, with the density error stored (tolerance mode);
// also p / rho*^2 for the pressure force.  Returns |err| (0 for a particle not updated)
// and, in a batch, its scene (-2 once that scene met the tolerance before iteration k).
template <int NB>
__device__ __forceinline__ float pred_density_one(const Params &P, float4 *pos, const float4 *__restrict__ xstar,
                                                  const unsigned *__restrict__ cell,
                                                  const unsigned *__restrict__ start,
                                                  const ListEntry *__restrict__ list,
                                                  const int *__restrict__ nbr, float *__restrict__ press,
                                                  float *__restrict__ rhostar, float *__restrict__ derr, int k,
                                                  float delta, int clamp_total, int i, int &sc) {
    float aerr = 0.f;
    sc = -1;   // batch: scene of particle i while its corrector still runs
    if (i < P.n && P.nscenes > 0) {
        sc = P.scene[i];
        if (scene_converged_before(P, sc, k)) sc = -2;
    }
    if (i < P.n && sc != -2) {
        const float4 xi = xstar[i];
        float sum = 1.f;   // the particle itself: W_std(0) / (315 / (64 pi h^3))
        tile_members<NB, true>(
            P, start, list, nbr, pos, cell[i], i, [&](unsigned j) { return __ldg(&xstar[j]); },
            [&](const float4 xj) {
                const float r2 = dist2(xi, xj);
                if (r2 < P.h2mz) {
                    const float x = 1.f - r2 * P.inv_h2;
                    sum += x * x * x;
                }
            });
        aerr = pred_density_end(P, pos, press, rhostar, derr, delta, clamp_total, i, sum);
    }
    return aerr;
}

// Per-scene maximum and sum of |err| of one warp's particles (lanes grouped by scene: one
// group per warp except at the boundaries between scenes).  All lanes call it.  Sums: FP32
// over the 32 lanes, FP64 from there on.
__device__ __forceinline__ void scene_error_reduce(const Params &P, int sc, float aerr, int k) {
    const int lane = threadIdx.x & 31;
    const double s = (double)warp_sum_f(aerr);
    const unsigned grp = __match_any_sync(0xffffffffu, sc);
    const unsigned gm = __reduce_max_sync(grp, __float_as_uint(aerr));
    if (sc >= 0) {
        if ((__ffs(grp) - 1) == lane && gm) atomicMax(&P.scene_st[sc].err_bits[k], gm);
        if (grp == 0xffffffffu) {
            if (lane == 0) atomicAdd(&P.scene_st[sc].err_sum[k], s);
        } else {
            atomicAdd(&P.scene_st[sc].err_sum[k], (double)aerr);
        }
    }
}

// Block reduction of max |err| (exact as bits of non-negative floats) and sum |err| into
// iteration k's totals: FP32 within a warp (at most 32 x particles-per-thread terms), FP64
// across warps and blocks.  All threads call it.
__device__ __forceinline__ void error_reduce(StepState *st, float amax, float asum, int k) {
    __shared__ unsigned smax[kMaxTile / 32];
    __shared__ double ssum[kMaxTile / 32];
    const unsigned m = warp_max_u(__float_as_uint(amax));
    const double s = (double)warp_sum_f(asum);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) { smax[wid] = m; ssum[wid] = s; }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned bm = 0;
        double bs = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) { bm = max(bm, smax[w]); bs += ssum[w]; }
        if (bm) atomicMax(&st->err_bits[k], bm);
        atomicAdd(&st->err_sum[k], bs);
    }
}

// k < 0: iteration index from the device (the graph's WHILE loop only runs unconverged
// iterations); k >= 0: host-launched sequence, skip after convergence.  Each pass of the loop
// advances the other's counter, which no block of its own launch reads: the predicted-density
// pass hands its iteration to the pressure-force pass, which starts the next one.
__device__ __forceinline__ bool density_iteration(const Params &P, StepState *st, int &k) {
    if (k < 0) {
        k = st->iter;
        if (blockIdx.x == 0 && threadIdx.x == 0) st->iter_pf = k;
        return true;
    }
    return !converged_before(P, st, k);
}

// Also the end of the loop (the break of ComputePressureForceAndIntegrate,
// pcisph_equations3.cpp:238-246): no further iteration once the density error of iteration k
// is below tolerance or k was the last allowed one.  The error is final before this launch,
// so one thread of it decides; a launch of its own for that cost 3 us an iteration.
__device__ __forceinline__ bool force_iteration(const Params &P, StepState *st, int &k, int max_it,
                                                cudaGraphConditionalHandle loop) {
    if (k < 0) {
        k = st->iter_pf;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            const bool done = (k >= max_it - 1) ||
                              fdv(__uint_as_float(st->err_bits[k]), P.target_density) < P.max_err_ratio;
            st->iter = k + 1;
            cudaGraphSetConditional(loop, done ? 0u : 1u);
        }
        return true;
    }
    return !converged_before(P, st, k);
}

// Work item w of the batch's list: the tile (segment of the scene found by binary search
// over the segment offsets).
__device__ __forceinline__ int worklist_tile(const Params &P, int w) {
    int lo = 0, hi = P.nscenes;   // wl_off[lo] <= w < wl_off[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(&P.wl_off[mid]) <= w) lo = mid;
        else hi = mid;
    }
    return __ldg(&P.wl_tile[lo]) + (w - __ldg(&P.wl_off[lo]));
}

// Number of work items, at most the number of tiles (of `slots` slots).
__device__ __forceinline__ int worklist_total(const Params &P, int slots) {
    const int tiles = (P.n + slots - 1) / slots;
    const int total = __ldg(&P.wl_off[P.nscenes]);
    return total < tiles ? total : tiles;
}

// Next work item of a persistent block (counter c; two shared slots alternate so that one
// barrier per item keeps the slot being read apart from the one being written).
__device__ __forceinline__ int worklist_next(int *ctr, int *slot, int &parity) {
    if (threadIdx.x == 0) slot[parity] = atomicAdd(ctr, 1);
    __syncthreads();
    const int w = slot[parity];
    parity ^= 1;
    return w;
}

// First slot of the block's tile of `slots` slots: the block's own, or with a batch work
// list (wl) the tile of work item blockIdx.x; -1 for a block past the list's end.
__device__ __forceinline__ int block_tile(const Params &P, int wl, int slots) {
    if (!wl) return tile_of_block(P, blockIdx.x, (P.n + slots - 1) / slots) * slots;
    if ((int)blockIdx.x >= worklist_total(P, slots)) return -1;
    return worklist_tile(P, blockIdx.x) * slots;
}

// One block per tile (all tiles, or the work list's) of PPT x blockDim slots; thread t
// takes slots t, t + blockDim, ... (PPT particles per thread).
template <int NB, int PPT, int MINB = kPdMinBlocks>
__global__ void __launch_bounds__(kMaxTile, MINB)
k_pred_density(Params P, float4 *pos, const float4 *__restrict__ xstar,
               const unsigned *__restrict__ cell, const unsigned *__restrict__ start,
               const ListEntry *__restrict__ list, const int *__restrict__ nbr, float *__restrict__ press,
               float *__restrict__ rhostar, float *__restrict__ derr, StepState *st, int k,
               float delta, int clamp_total, int wl) {
    if (!density_iteration(P, st, k)) return;
    const int s0 = block_tile(P, wl, PPT * blockDim.x);
    if (s0 < 0 || s0 >= P.n) return;
    float amax = 0.f, asum = 0.f;
#pragma unroll 1
    for (int u = 0; u < PPT; u++) {
        const int su = s0 + u * blockDim.x;
        int sc;
        const float aerr = pred_density_one<NB>(P, pos, xstar, cell, start, list, nbr, press, rhostar, derr,
                                                k, delta, clamp_total, su + threadIdx.x, sc);
        amax = fmaxf(amax, aerr);
        asum += aerr;
        if (P.nscenes > 0) scene_error_reduce(P, sc, aerr, k);
    }
    error_reduce(st, amax, asum, k);
}

// Batch: persistent blocks over the work list of the tiles whose scenes still run
// (launch_worklist), the same per-particle work as k_pred_density.
template <int NB>
__global__ void __launch_bounds__(kMaxTile, kPdWlMinBlocks)
k_pred_density_wl(Params P, float4 *pos, const float4 *__restrict__ xstar,
                  const unsigned *__restrict__ cell, const unsigned *__restrict__ start,
                  const ListEntry *__restrict__ list, const int *__restrict__ nbr, float *__restrict__ press,
                  float *__restrict__ rhostar, float *__restrict__ derr, StepState *st, int k,
                  float delta, int clamp_total) {
    if (!density_iteration(P, st, k)) return;
    __shared__ int slot[2];
    int parity = 0;
    const int total = worklist_total(P, blockDim.x);
    float amax = 0.f, asum = 0.f;   // this thread's particles (a few tiles): FP32 partial sum
    for (;;) {
        const int w = worklist_next(&P.wl_ctr[0], slot, parity);
        if (w >= total) break;
        const int s0 = worklist_tile(P, w) * blockDim.x;
        if (s0 < 0 || s0 >= P.n) continue;   // never for a list built by k_worklist
        int sc;
        const float aerr = pred_density_one<NB>(P, pos, xstar, cell, start, list, nbr, press, rhostar, derr,
                                                k, delta, clamp_total, s0 + threadIdx.x, sc);
        amax = fmaxf(amax, aerr);
        asum += aerr;
        scene_error_reduce(P, sc, aerr, k);
    }
    error_reduce(st, amax, asum, k);
}

// What follows a particle's pressure force fp: the next prediction, or with `last`
// AccumulateForcesFor + TimeIntegrationFor.
__device__ __forceinline__ void pressure_force_end(const Params &P, const float4 *__restrict__ vel, float4 *__restrict__ force,
                                                   float4 *__restrict__ pforce, float4 *__restrict__ xstar,
                                                   float4 *__restrict__ pos_out, float4 *__restrict__ vel_out, float dt,
                                                   float dt_over_m, int mode, bool last, int i, float4 pi, v3 fp,
                                                   unsigned &fbits, bool &bad) {
    pforce[i] = F4(fp);
    const v3 f = V(force[i]);
    if (last) {
        const v3 ft = vadd(f, fp);
        force[i] = F4(ft);
        v3 x = V(pi), v = V(vel[i]);
        integrate_particle(P, dt, ft, &x, &v);
        pos_out[i] = F4(x);
        vel_out[i] = F4(v);
        fbits = max(fbits, __float_as_uint(vlen(ft)));
        bad = bad || !finite_state(x, v);
    } else if (mode != 1) {
        v3 xs;
        predict_particle(P, dt, dt_over_m, f, fp, V(pi), V(vel[i]), &xs);
        xstar[i] = F4(xs);
    }
}

// PredictPressureForceFor (pcisph_equations3.cpp:114-155) of particle i at the current
// positions, then either the next prediction or AccumulateForcesFor + TimeIntegrationFor.
// `last`: iteration k ends the corrector (single scene); batches decide per scene.
template <int NB>
__device__ __forceinline__ void pressure_force_one(const Params &P, const float4 *__restrict__ pos,
                                                   const float4 *__restrict__ vel,
                                                   const unsigned *__restrict__ cell,
                                                   const unsigned *__restrict__ start,
                                                   const ListEntry *__restrict__ list,
                                                   const int *__restrict__ nbr, float4 *__restrict__ force,
                                                   float4 *__restrict__ pforce, float4 *__restrict__ xstar,
                                                   float4 *__restrict__ pos_out, float4 *__restrict__ vel_out,
                                                   int k, int max_it, float dt, float dt_over_m, int mode,
                                                   bool last, int i, unsigned &fbits, bool &bad) {
    bool active = i < P.n;
    if (active && P.nscenes > 0) {
        // batch: each scene stops at its own convergence
        const int sc = P.scene[i];
        active = !scene_converged_before(P, sc, k);
        last = mode == 0 && ((k == max_it - 1) ||
                             fdv(__uint_as_float(P.scene_st[sc].err_bits[k]), P.target_density) < P.max_err_ratio);
    }
    if (!active) return;
    const float4 pi = pos[i];
    const float ai = pi.w;   // p_i / rho*_i^2
    float tx = 0.f, ty = 0.f, tz = 0.f;
    const float kg = P.m2 * P.spiky_dw_c;
    tile_members<NB>(
        P, start, list, nbr, pos, cell[i], i, [&](unsigned j) { return __ldg(&pos[j]); },
        [&](const float4 pj) {   // pj.w = p_j / rho*_j^2
            const float r2 = dist2(pi, pj);
            const float inv_d = rsqrtf(r2);
            const float d = r2 > 0.f ? r2 * inv_d : 0.f;   // coincident particles: distance 0
            // IsWithinSpiky(d, h) and d > 0 && !IsZero(d)
            if (d - P.h <= -P.iz && d >= P.iz) {
                const float x = 1.f - d * P.inv_h;
                const float c = kg * (ai + pj.w) * x * x * inv_d;
                tx += (pj.x - pi.x) * c;
                ty += (pj.y - pi.y) * c;
                tz += (pj.z - pi.z) * c;
            }
        });
    pressure_force_end(P, vel, force, pforce, xstar, pos_out, vel_out, dt, dt_over_m, mode, last, i, pi,
                       V(-tx, -ty, -tz), fbits, bad);
}

__device__ __forceinline__ bool corrector_ends(const Params &P, const StepState *st, int k, int max_it, int mode) {
    return mode == 0 && ((k == max_it - 1) ||
                         fdv(__uint_as_float(st->err_bits[k]), P.target_density) < P.max_err_ratio);
}

template <int NB, int PPT, int MINB = kPfMinBlocks>
__global__ void __launch_bounds__(kMaxTile, MINB)
k_pressure_force(Params P, const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                 const unsigned *__restrict__ cell, const unsigned *__restrict__ start,
                 const ListEntry *__restrict__ list, const int *__restrict__ nbr, float4 *__restrict__ force,
                 float4 *__restrict__ pforce,
                 float4 *__restrict__ xstar, float4 *__restrict__ pos_out,
                 float4 *__restrict__ vel_out, StepState *st, int k, int max_it, float dt,
                 float dt_over_m, int mode, int wl, cudaGraphConditionalHandle loop) {
    if (!force_iteration(P, st, k, max_it, loop)) return;
    const bool last = corrector_ends(P, st, k, max_it, mode);
    const int s0 = block_tile(P, wl, PPT * blockDim.x);
    if (s0 < 0 || s0 >= P.n) return;
    unsigned fbits = 0;
    bool bad = false;   // integrated position or velocity not finite
#pragma unroll 1
    for (int u = 0; u < PPT; u++) {
        const int su = s0 + u * blockDim.x;
        pressure_force_one<NB>(P, pos, vel, cell, start, list, nbr, force, pforce, xstar, pos_out, vel_out,
                               k, max_it, dt, dt_over_m, mode, last, su + threadIdx.x, fbits, bad);
    }
    fbits = warp_max_u(fbits);
    if ((threadIdx.x & 31) == 0 && fbits) atomicMax(&st->max_force_bits, fbits);
    count_nonfinite(bad, st);
}

// Batch: persistent blocks over the same work list as k_pred_density_wl.
template <int NB>
__global__ void __launch_bounds__(kMaxTile, kPfWlMinBlocks)
k_pressure_force_wl(Params P, const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                    const unsigned *__restrict__ cell, const unsigned *__restrict__ start,
                    const ListEntry *__restrict__ list, const int *__restrict__ nbr, float4 *__restrict__ force,
                    float4 *__restrict__ pforce, float4 *__restrict__ xstar, float4 *__restrict__ pos_out,
                    float4 *__restrict__ vel_out, StepState *st, int k, int max_it, float dt, float dt_over_m,
                    int mode, cudaGraphConditionalHandle loop) {
    if (!force_iteration(P, st, k, max_it, loop)) return;
    __shared__ int slot[2];
    int parity = 0;
    const int total = worklist_total(P, blockDim.x);
    unsigned fbits = 0;
    bool bad = false;
    for (;;) {
        const int w = worklist_next(&P.wl_ctr[1], slot, parity);
        if (w >= total) break;
        const int s0 = worklist_tile(P, w) * blockDim.x;
        if (s0 < 0 || s0 >= P.n) continue;   // never for a list built by k_worklist
        pressure_force_one<NB>(P, pos, vel, cell, start, list, nbr, force, pforce, xstar, pos_out, vel_out, k,
                               max_it, dt, dt_over_m, mode, false, s0 + threadIdx.x, fbits, bad);
    }
    fbits = warp_max_u(fbits);
    if ((threadIdx.x & 31) == 0 && fbits) atomicMax(&st->max_force_bits, fbits);
    count_nonfinite(bad, st);
}

// Batch: first and last sorted slot of every scene (both arrays preset to 0x7f7f7f7f / -1).
// The layout keeps each scene's slots contiguous and the scenes in order (containers
// stacked along z, the slowest axis of the cell order, two empty cells apart).
__global__ void __launch_bounds__(kThreads)
k_scene_slots(Params P) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    const int s = P.scene[i];
    if (i == 0 || P.scene[i - 1] != s) atomicMin(&P.scene_first[s], i);
    if (i == P.n - 1 || P.scene[i + 1] != s) atomicMax(&P.scene_last[s], i);
}

// Exclusive block scan (sum, or max with identity INT_MIN) of one int per thread; *total
// gets the whole block's result.  All threads call it; sh holds 32 ints.
template <bool MAX>
__device__ __forceinline__ int block_scan_excl(int v, int *sh, int *total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
    const int id = MAX ? INT_MIN : 0;
    auto op = [](int a, int b) { return MAX ? (a > b ? a : b) : a + b; };
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x = op(x, y);
    }
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int t = lane < nw ? sh[lane] : id;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t = op(t, y);
        }
        sh[lane] = t;
    }
    __syncthreads();
    const int before = __shfl_up_sync(0xffffffffu, x, 1);
    const int r = op(wid > 0 ? sh[wid - 1] : id, lane > 0 ? before : id);
    *total = sh[nw - 1];
    __syncthreads();
    return r;
}

// Batch work list of corrector iteration k (k < 0: the device counter): for every scene
// whose corrector still runs, the segment of tiles (of `tile` slots) holding its slots,
// without the tiles an earlier segment already holds; a scene that met the tolerance gets
// an empty segment.  Resets the persistent passes' counters.  One block.
__global__ void __launch_bounds__(1024)
k_worklist(Params P, const StepState *st, int k, int tile) {
    __shared__ int sh[32];
    if (k < 0) k = st->iter;
    int carry_tile = -1;   // last tile of the segments so far
    int carry_off = 0;     // work items so far
    for (int c = 0; c < P.nscenes; c += blockDim.x) {
        const int s = c + threadIdx.x;
        int ta = 0, tb = -1;
        if (s < P.nscenes) {
            const int f = P.scene_first[s], l = P.scene_last[s];
            if (l >= f && l >= 0 && !scene_converged_before(P, s, k)) {
                ta = f / tile;
                tb = l / tile;
            }
        }
        int chunk_max, chunk_sum;
        const int before = block_scan_excl<true>(tb, sh, &chunk_max);
        const int prev = max(carry_tile, before);
        if (ta <= prev) ta = prev + 1;
        const int len = tb >= ta ? tb - ta + 1 : 0;
        const int off = block_scan_excl<false>(len, sh, &chunk_sum);
        if (s < P.nscenes) {
            P.wl_off[s] = carry_off + off;
            P.wl_tile[s] = ta;
        }
        carry_tile = max(carry_tile, chunk_max);
        carry_off += chunk_sum;
    }
    if (threadIdx.x == 0) {
        P.wl_off[P.nscenes] = carry_off;
        P.wl_ctr[0] = 0;
        P.wl_ctr[1] = 0;
    }
}

// The corrector's passes with G lanes per particle (see kGroup16), in the manner of
// k_sph_forces_group; single scenes only, since a batch's blocks walk tiles of its scenes.  A
// substep of 8,400 particles, 3 iterations: 98.7 -> 92.1 us; 12,144, 9 iterations: 201 -> 189; 18,252, 5
// iterations: 137 -> 133.  What is left of an iteration is two launches and the loop's condition.
template <int G>
__global__ void __launch_bounds__(kGroupThreads, 8)
k_pred_density_group(Params P, float4 *pos, const float4 *__restrict__ xstar, const unsigned *__restrict__ cell,
                     const unsigned *__restrict__ start, const ListEntry *__restrict__ list,
                     const int *__restrict__ nbr, float *__restrict__ press, float *__restrict__ rhostar,
                     float *__restrict__ derr, StepState *st, int k, float delta, int clamp_total) {
    if (!density_iteration(P, st, k)) return;
    constexpr int S = kGroupThreads / G, NB = 32 / G;
    __shared__ float term[kMaxList][S];   // x of the member's x^3; 0 outside the kernel, which adds nothing
    const int grp = threadIdx.x / G, lane = threadIdx.x & (G - 1);
    const int at = blockIdx.x * S + grp;
    if (at < P.n) {
        const float4 xi = xstar[at];
        const unsigned cw = cell[at];
        const int cnt = cw & kWide ? 0 : __ldg(&nbr[at]) - 1;
        const ListEntry *const l = list + at;
        for (int q0 = lane; q0 < cnt; q0 += NB * G) {
            unsigned j[NB];
#pragma unroll
            for (int u = 0; u < NB; u++) j[u] = q0 + u * G < cnt ? __ldg(l + (size_t)(q0 + u * G) * P.n) : (unsigned)at;
            float4 xj[NB];
#pragma unroll
            for (int u = 0; u < NB; u++) xj[u] = __ldg(&xstar[j[u]]);
#pragma unroll
            for (int u = 0; u < NB; u++) {
                const float r2 = dist2(xi, xj[u]);
                if (q0 + u * G < cnt) term[q0 + u * G][grp] = r2 < P.h2mz ? __fmaf_rn(-r2, P.inv_h2, 1.f) : 0.f;
            }
        }
    }
    __syncthreads();
    float aerr = 0.f;
    const int i = blockIdx.x * S + threadIdx.x;
    if (threadIdx.x < S && i < P.n) {
        const unsigned cw = cell[i];
        float sum = 1.f;   // the particle itself
        if (cw & kWide) {
            const float4 xi = xstar[i];
            tile_members<1>(P, start, list, nbr, pos, cw, i, [&](unsigned j) { return __ldg(&xstar[j]); },
                            [&](const float4 xj) {
                                const float r2 = dist2(xi, xj);
                                if (r2 < P.h2mz) {
                                    const float x = __fmaf_rn(-r2, P.inv_h2, 1.f);
                                    sum = __fmaf_rn(__fmul_rn(x, x), x, sum);
                                }
                            });
        } else {
            const int cnt = __ldg(&nbr[i]) - 1;
#pragma unroll 8
            for (int q = 0; q < cnt; q++) {
                const float x = term[q][threadIdx.x];
                sum = __fmaf_rn(__fmul_rn(x, x), x, sum);
            }
        }
        aerr = pred_density_end(P, pos, press, rhostar, derr, delta, clamp_total, i, sum);
    }
    error_reduce(st, aerr, aerr, k);
}

template <int G>
__global__ void __launch_bounds__(kGroupThreads, 8)
k_pressure_force_group(Params P, const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                       const unsigned *__restrict__ cell, const unsigned *__restrict__ start,
                       const ListEntry *__restrict__ list, const int *__restrict__ nbr, float4 *__restrict__ force,
                       float4 *__restrict__ pforce, float4 *__restrict__ xstar, float4 *__restrict__ pos_out,
                       float4 *__restrict__ vel_out, StepState *st, int k, int max_it, float dt, float dt_over_m,
                       int mode, cudaGraphConditionalHandle loop) {
    if (!force_iteration(P, st, k, max_it, loop)) return;
    const bool last = corrector_ends(P, st, k, max_it, mode);
    constexpr int S = kGroupThreads / G, NB = G == 4 ? 4 : 32 / G, kTerms = NB * G;
    __shared__ float4 term[kTerms][S];   // (dx, dy, dz, c): the member adds (dx, dy, dz) * c; (0, 0, 0, 0): nothing
    __shared__ float sums[3][S];
    const int grp = threadIdx.x / G, lane = threadIdx.x & (G - 1);
    const int at = blockIdx.x * S + grp;
    const bool live = at < P.n;
    const float4 pa = pos[live ? at : P.n - 1];
    const unsigned ca = cell[live ? at : P.n - 1];
    const int cnt = live && !(ca & kWide) ? __ldg(&nbr[at]) - 1 : 0;
    const int longest = __reduce_max_sync(0xffffffffu, cnt);
    const ListEntry *const l = list + (live ? at : 0);
    const float kg = P.m2 * P.spiky_dw_c;
    const int dim = min(lane, 2);
    float acc = 0.f;
    for (int q0 = 0; q0 < longest; q0 += kTerms) {
        unsigned j[NB];
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const int q = q0 + u * G + lane;
            j[u] = q < cnt ? __ldg(l + (size_t)q * P.n) : 0u;
        }
        float4 pj[NB];
#pragma unroll
        for (int u = 0; u < NB; u++) pj[u] = __ldg(&pos[j[u]]);
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const float r2 = dist2(pa, pj[u]);
            const float inv_d = rsqrtf(r2);
            const float d = r2 > 0.f ? r2 * inv_d : 0.f;   // coincident particles: distance 0
            const float x = 1.f - d * P.inv_h;
            const float c = kg * (pa.w + pj[u].w) * x * x * inv_d;
            const bool in = d - P.h <= -P.iz && d >= P.iz;
            term[u * G + lane][grp] = in ? make_float4(pj[u].x - pa.x, pj[u].y - pa.y, pj[u].z - pa.z, c)
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncwarp();
        const float *e = reinterpret_cast<const float *>(&term[0][grp]);
        const int some = min(cnt - q0, kTerms);
#pragma unroll 8
        for (int q = 0; q < some; q++, e += 4 * S) acc = __fmaf_rn(e[dim], e[3], acc);
        __syncwarp();
    }
    if (lane < 3) sums[lane][grp] = acc;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const int i = blockIdx.x * S + threadIdx.x;
    unsigned fbits = 0;
    bool bad = false;
    if (threadIdx.x < S && i < P.n) {
        if (cell[i] & kWide) {
            pressure_force_one<1>(P, pos, vel, cell, start, list, nbr, force, pforce, xstar, pos_out, vel_out, k, max_it,
                                  dt, dt_over_m, mode, last, i, fbits, bad);
        } else {
            const v3 fp = V(-sums[0][threadIdx.x], -sums[1][threadIdx.x], -sums[2][threadIdx.x]);
            pressure_force_end(P, vel, force, pforce, xstar, pos_out, vel_out, dt, dt_over_m, mode, last, i, pos[i], fp,
                               fbits, bad);
        }
    }
    fbits = warp_max_u(fbits);
    if (threadIdx.x == 0 && fbits) atomicMax(&st->max_force_bits, fbits);
    count_nonfinite(bad, st);
}

// A member's terms in the SPH force pass.
struct SphPair {
    float dx, dy, dz, c;      // the pressure force's terms are (dx, dy, dz) * c
    float dvx, dvy, dvz, w;   // the viscosity's (dvx, dvy, dvz) * w
    bool near, apart;         // inside the kernels; and not coincident
    __device__ __forceinline__ SphPair(const Params &P, float4 pi, float4 vi, float4 pj, float4 vj, float ai, float kg,
                                       float kv) {
        const float r2 = dist2(pi, pj);
        const float inv_d = rsqrtf(r2);
        const float d = r2 > 0.f ? r2 * inv_d : 0.f;   // coincident particles: distance 0
        near = d - P.h <= -P.iz;
        apart = d >= P.iz;
        const float x = 1.f - d * P.inv_h;
        c = kg * (ai + pj.w) * x * x * inv_d;
        w = kv * x * vj.w;   // vj.w = 1 / rho_j
        dx = pj.x - pi.x;
        dy = pj.y - pi.y;
        dz = pj.z - pi.z;
        dvx = vj.x - vi.x;
        dvy = vj.y - vi.y;
        dvz = vj.z - vi.z;
    }
};

// What the force passes add a member to: t the pressure force's sum, f the rest.
struct SphForce {
    v3 f, t;
    __device__ __forceinline__ void add(const SphPair &a) {
        if (a.near) {
            if (a.apart) {
                t.x = __fmaf_rn(a.dx, a.c, t.x);
                t.y = __fmaf_rn(a.dy, a.c, t.y);
                t.z = __fmaf_rn(a.dz, a.c, t.z);
            }
            f.x = __fmaf_rn(a.dvx, a.w, f.x);
            f.y = __fmaf_rn(a.dvy, a.w, f.y);
            f.z = __fmaf_rn(a.dvz, a.w, f.z);
        }
    }
};

// ComputeAllForcesFor (sph_equations3.cpp:184-278, extended = 0) in Jacobi order: the
// reference integrates each particle inside the force loop (:277), racing with its
// neighbours' reads; here all forces read the step-start state and the integrated
// state goes to the other buffer.
template <int NB>
__global__ void __launch_bounds__(kMaxTile)
k_sph_forces(Params P, const float4 *__restrict__ pos, const float4 *__restrict__ vel,
             const unsigned *__restrict__ cell, const unsigned *__restrict__ start,
             const ListEntry *__restrict__ list, const int *__restrict__ nbr, float4 *__restrict__ force,
             float4 *__restrict__ pos_out, float4 *__restrict__ vel_out, StepState *st, float dt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned fbits = 0;
    bool bad = false;   // integrated position or velocity not finite
    if (i < P.n) {
        const float4 pi = pos[i];
        const float4 vi = vel[i];
        const float ai = pi.w;   // p_i / rho_i^2
        SphForce a{V(P.mass * P.gx - P.drag * vi.x, P.mass * P.gy - P.drag * vi.y, P.mass * P.gz - P.drag * vi.z),
                   V(0.f, 0.f, 0.f)};
        const float kg = P.m2 * P.spiky_dw_c;
        const float kv = P.visc_m2 * P.spiky_d2w_c;
        tile_members<NB>(
            P, start, list, nbr, pos, cell[i], i,
            [&](unsigned j) { return PosVel{__ldg(&pos[j]), __ldg(&vel[j])}; },
            [&](const PosVel &nb) { a.add(SphPair(P, pi, vi, nb.p, nb.v, ai, kg, kv)); });
        const v3 f = V(a.f.x - a.t.x, a.f.y - a.t.y, a.f.z - a.t.z);
        force[i] = F4(f);
        v3 x = V(pi), v = V(vi);
        integrate_particle(P, dt, f, &x, &v);
        pos_out[i] = F4(x);
        vel_out[i] = F4(v);
        fbits = __float_as_uint(vlen(f));
        bad = !finite_state(x, v);
    }
    fbits = warp_max_u(fbits);
    if ((threadIdx.x & 31) == 0 && fbits) atomicMax(&st->max_force_bits, fbits);
    count_nonfinite(bad, st);
}

// The same with G lanes per particle (see kGroup16): the lanes take every G-th member and leave its
// terms in shared memory, 4 G members at a time, and each of the six sums is added up over them in
// list order by a lane, as k_sph_forces adds them.  One warp then integrates the block's particles.  Blocks
// of 16 KB and 64 registers: with all 64 members' terms in shared memory, 6 blocks an SM, 16,384
// particles took 18 us, so 14 (four lanes 12).  1,287 particles: 12.3 -> 8.2 us.
template <int G>
__global__ void __launch_bounds__(kGroupThreads, 8)
k_sph_forces_group(Params P, const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                   const unsigned *__restrict__ cell, const unsigned *__restrict__ start,
                   const ListEntry *__restrict__ list, const int *__restrict__ nbr, float4 *__restrict__ force,
                   float4 *__restrict__ pos_out, float4 *__restrict__ vel_out, StepState *st, float dt) {
    constexpr int S = kGroupThreads / G;   // particles of a block
    constexpr int NB = 4, kGroupTerms = NB * G;
    __shared__ float4 term[2][kGroupTerms][S];   // (dx, dy, dz, c), (dvx, dvy, dvz, w)
    __shared__ float sums[6][S];
    constexpr unsigned full = 0xffffffffu, group = (1u << G) - 1u;
    const int grp = threadIdx.x / G, lane = threadIdx.x & (G - 1);
    const int shift = threadIdx.x & 31 & ~(G - 1);
    const bool live = blockIdx.x * S + grp < P.n;
    const int i = live ? blockIdx.x * S + grp : P.n - 1;
    const float4 pi = pos[i];
    const float4 vi = vel[i];
    const float ai = pi.w;
    const v3 f0 = V(P.mass * P.gx - P.drag * vi.x, P.mass * P.gy - P.drag * vi.y, P.mass * P.gz - P.drag * vi.z);
    const float kg = P.m2 * P.spiky_dw_c;
    const float kv = P.visc_m2 * P.spiky_d2w_c;
    const unsigned cw = cell[i];
    const bool wide = (cw & kWide) != 0;
    const int cnt = live && !wide ? __ldg(&nbr[i]) - 1 : 0;
    const int longest = __reduce_max_sync(full, cnt);
    const ListEntry *const l = list + i;
    // the six sums: with eight lanes t in lanes 0 .. 2 and f in 3 .. 5, with four both in 0 .. 2
    // (the lanes left over along with the last)
    constexpr int per = G >= 6 ? 1 : 2;
    const int k = per == 2 ? min(lane, 2) : lane < 3 ? lane : min(lane, 5) - 3;
    const bool is_f = per == 1 && lane >= 3;
    const float fk = k == 0 ? f0.x : k == 1 ? f0.y : f0.z;
    float acc[per];
    acc[0] = is_f ? fk : 0.f;
    if (per == 2) acc[per - 1] = fk;
    const float *const e0 = reinterpret_cast<const float *>(&term[is_f ? 1 : 0][0][grp]);
    for (int q0 = 0; q0 < longest; q0 += kGroupTerms) {
        unsigned j[NB];
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const int q = q0 + u * G + lane;
            j[u] = q < cnt ? __ldg(l + (size_t)q * P.n) : (unsigned)i;
        }
        PosVel nb[NB];
#pragma unroll
        for (int u = 0; u < NB; u++) nb[u] = PosVel{__ldg(&pos[j[u]]), __ldg(&vel[j[u]])};
        unsigned near = 0, apart = 0;   // the group's members with terms
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const int q = u * G + lane;
            const SphPair a(P, pi, vi, nb[u].p, nb[u].v, ai, kg, kv);
            const bool in = q0 + q < cnt && a.near;
            if (in) {
                term[0][q][grp] = make_float4(a.dx, a.dy, a.dz, a.c);
                term[1][q][grp] = make_float4(a.dvx, a.dvy, a.dvz, a.w);
            }
            near |= ((__ballot_sync(full, in) >> shift) & group) << (u * G);
            apart |= ((__ballot_sync(full, in && a.apart) >> shift) & group) << (u * G);
        }
        __syncwarp();
        const unsigned take = is_f ? near : apart;
        const float *e = e0;
        const int some = min(cnt - q0, kGroupTerms);
#pragma unroll 4
        for (int q = 0; q < some; q++, e += 4 * S) {
            if ((take >> q) & 1u) acc[0] = __fmaf_rn(e[k], e[3], acc[0]);
            if (per == 2 && ((near >> q) & 1u))
                acc[per - 1] = __fmaf_rn(e[4 * kGroupTerms * S + k], e[4 * kGroupTerms * S + 3], acc[per - 1]);
        }
        __syncwarp();
    }
    if (per == 1 ? lane < 6 : lane < 3) {
        sums[lane][grp] = acc[0];
        if (per == 2) sums[3 + lane][grp] = acc[per - 1];
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    // the first warp: a lane per particle
    const int at = blockIdx.x * S + threadIdx.x;
    unsigned fbits = 0;
    bool bad = false;
    if (threadIdx.x < S && at < P.n) {
        const float4 pm = pos[at], vm = vel[at];
        const unsigned cm = cell[at];
        const int t = threadIdx.x;
        v3 f = V(sums[3][t] - sums[0][t], sums[4][t] - sums[1][t], sums[5][t] - sums[2][t]);
        if (cm & kWide) {
            SphForce a{V(P.mass * P.gx - P.drag * vm.x, P.mass * P.gy - P.drag * vm.y, P.mass * P.gz - P.drag * vm.z),
                       V(0.f, 0.f, 0.f)};
            tile_members<1>(P, start, list, nbr, pos, cm, at,
                            [&](unsigned j) { return PosVel{__ldg(&pos[j]), __ldg(&vel[j])}; },
                            [&](const PosVel &nb) { a.add(SphPair(P, pm, vm, nb.p, nb.v, pm.w, kg, kv)); });
            f = V(a.f.x - a.t.x, a.f.y - a.t.y, a.f.z - a.t.z);
        }
        force[at] = F4(f);
        v3 x = V(pm), v = V(vm);
        integrate_particle(P, dt, f, &x, &v);
        pos_out[at] = F4(x);
        vel_out[at] = F4(v);
        fbits = __float_as_uint(vlen(f));
        bad = !finite_state(x, v);
    }
    fbits = warp_max_u(fbits);
    if (threadIdx.x == 0 && fbits) atomicMax(&st->max_force_bits, fbits);
    count_nonfinite(bad, st);
}

// AccumulateForcesFor + TimeIntegrationFor (AccumulateAndIntegrateGPU,
// pcisph_equations3.cpp:179-212): F += Fp, then integrate into the other buffer.
__global__ void __launch_bounds__(kThreads)
k_accumulate_integrate(Params P, const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                       float4 *__restrict__ force, const float4 *__restrict__ pforce,
                       float4 *__restrict__ pos_out, float4 *__restrict__ vel_out, float dt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    const v3 ft = vadd(V(force[i]), V(pforce[i]));
    force[i] = F4(ft);
    v3 x = V(pos[i]), v = V(vel[i]);
    integrate_particle(P, dt, ft, &x, &v);
    pos_out[i] = F4(x);
    vel_out[i] = F4(v);
}

// TimeIntegrationFor over all particles (TimeIntegrationGPU, sph_equations3.cpp:622-634)
__global__ void __launch_bounds__(kThreads)
k_integrate(Params P, const float4 *__restrict__ pos, const float4 *__restrict__ vel,
            const float4 *__restrict__ force, float4 *__restrict__ pos_out,
            float4 *__restrict__ vel_out, float dt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    v3 x = V(pos[i]), v = V(vel[i]);
    integrate_particle(P, dt, V(force[i]), &x, &v);
    pos_out[i] = F4(x);
    vel_out[i] = F4(v);
}

// ComputePseudoViscosityAggregationKernelFor (sph_equations3.cpp:341-371): membership
// from the step-start positions (the bucket), values at the integrated state.
__global__ void __launch_bounds__(kMaxTile)
k_pv_aggregate(Params P, const float4 *__restrict__ pos_old, const float4 *__restrict__ pos,
               const float4 *__restrict__ vel, const float *__restrict__ inv_rho,
               const unsigned *__restrict__ cell, const unsigned *__restrict__ start,
               const ListEntry *__restrict__ list, const int *__restrict__ nbr, float4 *__restrict__ smoothed) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    const float4 pi = pos[i];
    // the particle itself (distance 0): W_spiky(0) m / rho_i
    const float w0 = P.mass * __ldg(&inv_rho[i]) * P.spiky_w_c;
    const float4 v0 = vel[i];
    float ws = w0, sx = w0 * v0.x, sy = w0 * v0.y, sz = w0 * v0.z;
    tile_members(
        P, start, list, nbr, pos_old, cell[i], i, [&](unsigned j) { return j; },
        [&](unsigned j) {
            const float4 pj = __ldg(&pos[j]);
            const float d = sqrtf(dist2(pi, pj));
            if (d - P.h <= -P.iz) {
                const float x = 1.f - d * P.inv_h;
                const float wj = P.mass * __ldg(&inv_rho[j]) * (P.spiky_w_c * x * x * x);
                const float4 vj = __ldg(&vel[j]);
                ws += wj;
                sx += wj * vj.x;
                sy += wj * vj.y;
                sz += wj * vj.z;
            }
        });
    if (ws > 0.f) {
        const float inv = 1.f / ws;
        sx *= inv; sy *= inv; sz *= inv;
    }
    smoothed[i] = make_float4(sx, sy, sz, 0.f);
}

// ComputePseudoViscosityInterpolationKernelFor (sph_equations3.cpp:373-382)
__global__ void k_pv_interpolate(int n, float4 *__restrict__ vel, const float4 *__restrict__ smoothed,
                                 float t) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 v = vel[i], s = smoothed[i];
    const float a = 1.f - t;
    vel[i] = make_float4(v.x * a + s.x * t, v.y * a + s.y * t, v.z * a + s.z * t, 0.f);
}

// Neighbour sets of the last density pass in caller order (bbg_neighbor_lists): every
// particle whose original id lies in [a, b) writes its members other than itself, as
// original ids in visit order (at most maxm of them, -1 after the last), into row id - a of
// out, and its full member count into counts[id - a].  pos0 holds the positions of that
// density pass (wide particles re-test their candidates there).
__global__ void __launch_bounds__(kThreads)
k_export_members(Params P, const unsigned *__restrict__ cell, const unsigned *__restrict__ start,
                 const ListEntry *__restrict__ list, const int *__restrict__ nbr,
                 const float4 *__restrict__ pos0, const int *__restrict__ pid, int a, int b, int maxm,
                 int *__restrict__ counts, int *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    const int id = pid[i];
    if (id < a || id >= b) return;
    int *row = out + (size_t)(id - a) * (size_t)maxm;
    int c = 0;
    tile_members<1>(P, start, list, nbr, pos0, cell[i], i, [&](unsigned j) { return j; },
                    [&](unsigned j) {
                        if (c < maxm) row[c] = pid[j];
                        c++;
                    });
    for (int q = c; q < maxm; q++) row[q] = -1;
    counts[id - a] = c;
}

void launch_export_members(const Params &P, const DevBufs &B, int buf, int pid_buf, int a, int b, int maxm,
                           int *counts, int *out, cudaStream_t s) {
    k_export_members<<<blocks_for(P.n, kThreads), kThreads, 0, s>>>(P, B.cell, B.start, B.list, B.nbr, B.pos[buf],
                                                                    B.pid[pid_buf], a, b, maxm, counts, out);
}

void launch_density(const Params &P, const DevBufs &B, int buf, int compute_pressure, cudaStream_t s, bool recorded) {
    BBG_PBEGIN(B, KID_DENSITY, s, -1);
    const int t = B.tune.block;
#define DENSITY_GROUP(G)                                                                          \
    k_density_group<G><<<blocks_for(P.n, kGroupThreads / G), kGroupThreads, 0, s>>>(              \
        P, B.pos[buf], B.vel[buf], B.cell, B.start, B.rho, B.inv_rho, B.press, B.nbr, B.list,     \
        compute_pressure, B.st)
    if (P.n <= kGroup16) {
        DENSITY_GROUP(16);
    } else if (P.n <= kGroup8) {
        DENSITY_GROUP(8);
    } else {
        if (!recorded)
            k_filter_records<<<blocks_for(P.n, kThreads), kThreads, 0, s>>>(P, B.pos[buf], B.cell,
                                                                            reinterpret_cast<__half *>(B.frec));
        const auto density = P.n <= kFew ? k_density_mask<true> : k_density_mask<false>;
        density<<<blocks_for(P.n, t), t, sizeof(uint2) * kMasks * (size_t)t, s>>>(
            P, B.pos[buf], B.vel[buf], B.cell, B.start, B.frec, B.rho, B.inv_rho, B.press, B.nbr, B.list,
            compute_pressure, B.st);
    }
#undef DENSITY_GROUP
    if (P.nscenes > 0 && P.n > 0) {
        // batch: each scene's slot range (the scene of every slot was set just above)
        cudaMemsetAsync(P.scene_first, 0x7f, sizeof(int) * (size_t)P.nscenes, s);
        cudaMemsetAsync(P.scene_last, 0xff, sizeof(int) * (size_t)P.nscenes, s);
        k_scene_slots<<<blocks_for(P.n, kThreads), kThreads, 0, s>>>(P);
    }
    BBG_PEND(B, s);
}

// Blocks of a member-walking pass over tiles of `slots` slots, in the tuned tile order
// (Params::tile_sms of the returned parameters).
static int tiled_grid(const Params &P, const DevBufs &B, int slots, Params *Q) {
    *Q = P;
    Q->tile_sms = 0;
    const int tiles = blocks_for(P.n, slots);
    if (B.tune.tile_order != 1 || P.nscenes > 0) return tiles;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) return tiles;
    Q->tile_sms = sms;
    return sms * ((tiles + sms - 1) / sms);
}

template <bool DIV, bool WARM>
static void non_pressure_nb(const Params &P0, const DevBufs &B, int buf, int predict, float dt,
                            float dt_over_m, cudaStream_t s, float *divsum) {
    const int t = B.tune.block;
    Params P;
    const int grid = tiled_grid(P0, B, t, &P);
#define NP_LAUNCH(...)                                                                       \
    k_non_pressure<DIV, WARM, __VA_ARGS__><<<grid, t, 0, s>>>(                                        \
        P, B.pos[buf], B.vel[buf], B.cell, B.start, B.list, B.nbr, B.force, B.xstar, B.pforce, \
        B.press, divsum, predict, dt, dt_over_m)
    if (P.n <= kFew) NP_LAUNCH(kFewBatchPosVel, 1);
    else switch (B.tune.batch_np) {
        case 2: NP_LAUNCH(2); break;
        case 8: NP_LAUNCH(8); break;
        default: NP_LAUNCH(4); break;
    }
#undef NP_LAUNCH
}

void launch_non_pressure(const Params &P, const DevBufs &B, int buf, int predict, float dt,
                         float dt_over_m, cudaStream_t s, float *divsum, bool warm) {
    BBG_PBEGIN(B, KID_NON_PRESSURE, s, -1);
    if (divsum) {
        if (warm) non_pressure_nb<true, true>(P, B, buf, predict, dt, dt_over_m, s, divsum);
        else non_pressure_nb<true, false>(P, B, buf, predict, dt, dt_over_m, s, divsum);
    } else {
        if (warm) non_pressure_nb<false, true>(P, B, buf, predict, dt, dt_over_m, s, nullptr);
        else non_pressure_nb<false, false>(P, B, buf, predict, dt, dt_over_m, s, nullptr);
    }
    BBG_PEND(B, s);
}

void launch_predict_first(const Params &P, const DevBufs &B, int buf, int is_first, float dt,
                          float dt_over_m, cudaStream_t s) {
    BBG_PBEGIN(B, KID_PREDICT_FIRST, s, -1);
    k_predict_first<<<blocks_for(P.n, kThreads), kThreads, 0, s>>>(
        P, B.pos[buf], B.vel[buf], B.force, B.xstar, B.pforce, B.press, B.rhostar, B.rho, B.derr,
        is_first, dt, dt_over_m);
    BBG_PEND(B, s);
}

// Resident blocks of a persistent kernel: every SM filled to the kernel's occupancy.
template <class K>
static int persistent_blocks(K kernel, int threads) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, 0);
    return (sms > 0 ? sms : 1) * (per > 0 ? per : 1);
}

template <int NB>
static int pd_grid(int t) { return persistent_blocks(k_pred_density_wl<NB>, t); }
template <int NB>
static int pf_grid(int t) { return persistent_blocks(k_pressure_force_wl<NB>, t); }

void update_worklist_grid(DevBufs &B) {
    const int t = B.tune.block;
    B.tune.wl_grid_pd = B.tune.batch_pd == 2 ? pd_grid<2>(t) : B.tune.batch_pd == 8 ? pd_grid<8>(t) : pd_grid<4>(t);
    B.tune.wl_grid_pf = B.tune.batch_pf == 2 ? pf_grid<2>(t) : B.tune.batch_pf == 8 ? pf_grid<8>(t) : pf_grid<4>(t);
}

// Particles per thread of the per-tile corrector passes (few particles: one).
static int corrector_ppt(const Params &P, const DevBufs &B) { return B.tune.ppt == 2 && P.n > kFew ? 2 : 1; }

// Slots per tile of the corrector passes: the block, times the particles per thread for
// the per-tile kernels.
static int corrector_tile(const Params &P, const DevBufs &B) {
    return B.tune.block * (B.tune.worklist == 2 ? 1 : corrector_ppt(P, B));
}

void launch_worklist(const Params &P, const DevBufs &B, int k, cudaStream_t s) {
    k_worklist<<<1, 1024, 0, s>>>(P, B.st, k, corrector_tile(P, B));
}

void launch_pred_density(const Params &P, const DevBufs &B, int buf, int k, float delta,
                         cudaStream_t s, int clamp_total) {
    BBG_PBEGIN(B, KID_PRED_DENSITY, s, k);
    const int t = B.tune.block;
    const int wl = P.nscenes > 0 ? B.tune.worklist : 0;
    if (wl) launch_worklist(P, B, k, s);   // batch: the tiles of the scenes still running
    if (wl == 2) {
        // persistent blocks over the work list
#define PD_LAUNCH(NB)                                                                               \
    k_pred_density_wl<NB><<<B.tune.wl_grid_pd > 0 ? B.tune.wl_grid_pd : pd_grid<NB>(t), t, 0, s>>>(  \
        P, B.pos[buf], B.xstar, B.cell, B.start, B.list, B.nbr, B.press, B.rhostar, B.derr, B.st, k, \
        delta, clamp_total)
        switch (B.tune.batch_pd) {
            case 2: PD_LAUNCH(2); break;
            case 8: PD_LAUNCH(8); break;
            default: PD_LAUNCH(4); break;
        }
#undef PD_LAUNCH
    } else {
        const int ppt = corrector_ppt(P, B);
        Params Q;
        const int grid = wl ? blocks_for(P.n, t * ppt) : tiled_grid(P, B, t * ppt, &Q);
        if (wl) Q = P;
#define PD_LAUNCH(...)                                                                            \
    k_pred_density<__VA_ARGS__><<<grid, t, 0, s>>>(Q, B.pos[buf], B.xstar, B.cell, B.start, B.list, B.nbr, \
                                               B.press, B.rhostar, B.derr, B.st, k, delta, clamp_total, wl)
#define PD_GROUP(G)                                                                                       \
    k_pred_density_group<G><<<blocks_for(P.n, kGroupThreads / G), kGroupThreads, 0, s>>>(                  \
        P, B.pos[buf], B.xstar, B.cell, B.start, B.list, B.nbr, B.press, B.rhostar, B.derr, B.st, k, delta, \
        clamp_total)
        if (P.n <= kGroup16 && P.nscenes == 0) PD_GROUP(8);
        else if (P.n <= kGroup8 && P.nscenes == 0) PD_GROUP(4);
        else if (P.n <= kFew) PD_LAUNCH(kFewBatch, 1, 1);
#undef PD_GROUP
        else switch (B.tune.batch_pd * 10 + ppt) {
            case 21: PD_LAUNCH(2, 1); break;
            case 81: PD_LAUNCH(8, 1); break;
            case 22: PD_LAUNCH(2, 2); break;
            case 42: PD_LAUNCH(4, 2); break;
            case 82: PD_LAUNCH(8, 2); break;
            default: PD_LAUNCH(4, 1); break;
        }
#undef PD_LAUNCH
    }
    BBG_PEND(B, s);
}

void launch_warm_start(const Params &P, const DevBufs &B, int buf, float scale, cudaStream_t s) {
    k_warm_start<<<blocks_for(P.n, kThreads), kThreads, 0, s>>>(P.n, B.pos[buf], B.rho, B.pprev,
                                                                B.press, B.rhostar, B.derr, scale);
}

void launch_pack_acoef(const Params &P, const DevBufs &B, int buf, cudaStream_t s) {
    k_pack_acoef<<<blocks_for(P.n, kThreads), kThreads, 0, s>>>(P.n, B.pos[buf], B.press, B.rhostar);
}

void launch_pressure_force(const Params &P, const DevBufs &B, int buf, int k, int max_it, float dt,
                           float dt_over_m, cudaStream_t s, int mode, cudaGraphConditionalHandle loop) {
    BBG_PBEGIN(B, KID_PRESSURE_FORCE, s, k);
    const int t = B.tune.block;
    const int wl = P.nscenes > 0 ? B.tune.worklist : 0;
    // batch: the work list launch_pred_density built for iteration k (built here when the
    // pass runs on its own)
    if (wl && mode == 1) launch_worklist(P, B, k, s);
    if (wl == 2) {
#define PF_LAUNCH(NB)                                                                                   \
    k_pressure_force_wl<NB><<<B.tune.wl_grid_pf > 0 ? B.tune.wl_grid_pf : pf_grid<NB>(t), t, 0, s>>>(    \
        P, B.pos[buf], B.vel[buf], B.cell, B.start, B.list, B.nbr, B.force, B.pforce, B.xstar,           \
        B.pos[1 - buf], B.vel[1 - buf], B.st, k, max_it, dt, dt_over_m, mode, loop)
        switch (B.tune.batch_pf) {
            case 2: PF_LAUNCH(2); break;
            case 8: PF_LAUNCH(8); break;
            default: PF_LAUNCH(4); break;
        }
#undef PF_LAUNCH
    } else {
        const int ppt = corrector_ppt(P, B);
        Params Q;
        const int grid = wl ? blocks_for(P.n, t * ppt) : tiled_grid(P, B, t * ppt, &Q);
        if (wl) Q = P;
#define PF_LAUNCH(...)                                                                                 \
    k_pressure_force<__VA_ARGS__><<<grid, t, 0, s>>>(                                                       \
        Q, B.pos[buf], B.vel[buf], B.cell, B.start, B.list, B.nbr, B.force, B.pforce, B.xstar,           \
        B.pos[1 - buf], B.vel[1 - buf], B.st, k, max_it, dt, dt_over_m, mode, wl, loop)
#define PF_GROUP(G)                                                                                      \
    k_pressure_force_group<G><<<blocks_for(P.n, kGroupThreads / G), kGroupThreads, 0, s>>>(                \
        P, B.pos[buf], B.vel[buf], B.cell, B.start, B.list, B.nbr, B.force, B.pforce, B.xstar,             \
        B.pos[1 - buf], B.vel[1 - buf], B.st, k, max_it, dt, dt_over_m, mode, loop)
        if (P.n <= kGroup16 && P.nscenes == 0) PF_GROUP(8);
        else if (P.n <= kGroup8 && P.nscenes == 0) PF_GROUP(4);
        else if (P.n <= kFew) PF_LAUNCH(kFewBatch, 1, 1);
#undef PF_GROUP
        else switch (B.tune.batch_pf * 10 + ppt) {
            case 21: PF_LAUNCH(2, 1); break;
            case 81: PF_LAUNCH(8, 1); break;
            case 22: PF_LAUNCH(2, 2); break;
            case 42: PF_LAUNCH(4, 2); break;
            case 82: PF_LAUNCH(8, 2); break;
            default: PF_LAUNCH(4, 1); break;
        }
#undef PF_LAUNCH
    }
    BBG_PEND(B, s);
}

void launch_sph_forces(const Params &P, const DevBufs &B, int buf, float dt, cudaStream_t s) {
    BBG_PBEGIN(B, KID_SPH_FORCES, s, -1);
    const int lanes = P.n <= kGroup16 ? 8 : P.n <= kGroup8 ? 4 : 1, t = lanes > 1 ? kGroupThreads : B.tune.block;
    const auto forces = lanes == 8    ? k_sph_forces_group<8>
                        : lanes == 4  ? k_sph_forces_group<4>
                        : P.n <= kFew ? k_sph_forces<kFewBatchPosVel>
                                      : k_sph_forces<(kGatherBatch < 4 ? kGatherBatch : 4)>;
    forces<<<blocks_for(P.n, t / lanes), t, 0, s>>>(
        P, B.pos[buf], B.vel[buf], B.cell, B.start, B.list, B.nbr, B.force, B.pos[1 - buf],
        B.vel[1 - buf], B.st, dt);
    BBG_PEND(B, s);
}

void launch_accumulate_integrate(const Params &P, const DevBufs &B, int buf, float dt,
                                 cudaStream_t s) {
    BBG_PBEGIN(B, KID_INTEGRATE, s, -1);
    k_accumulate_integrate<<<blocks_for(P.n, kThreads), kThreads, 0, s>>>(
        P, B.pos[buf], B.vel[buf], B.force, B.pforce, B.pos[1 - buf], B.vel[1 - buf], dt);
    BBG_PEND(B, s);
}

void launch_integrate(const Params &P, const DevBufs &B, int buf, float dt, cudaStream_t s) {
    BBG_PBEGIN(B, KID_INTEGRATE, s, -1);
    k_integrate<<<blocks_for(P.n, kThreads), kThreads, 0, s>>>(P, B.pos[buf], B.vel[buf], B.force,
                                                               B.pos[1 - buf], B.vel[1 - buf], dt);
    BBG_PEND(B, s);
}

// FP64 totals of the particle state: mass, kinetic energy, potential energy in the constant
// gravity field and momentum.  One partial row per block, summed by the host in block order,
// so the totals do not depend on scheduling.
constexpr int kEnergyBlocks = 1024;
__global__ void __launch_bounds__(kThreads)
k_energy(int n, const float4 *__restrict__ pos, const float4 *__restrict__ vel, double mass, double gx, double gy,
         double gz, double *__restrict__ partial) {
    double acc[kEnergyTerms] = {0, 0, 0, 0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 p = pos[i], v = vel[i];
        const double vx = v.x, vy = v.y, vz = v.z;
        acc[0] += mass;
        acc[1] += 0.5 * mass * (vx * vx + vy * vy + vz * vz);
        acc[2] -= mass * (gx * (double)p.x + gy * (double)p.y + gz * (double)p.z);
        acc[3] += mass * vx;
        acc[4] += mass * vy;
        acc[5] += mass * vz;
    }
    __shared__ double red[kThreads / 32][kEnergyTerms];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int t = 0; t < kEnergyTerms; t++) {
        const double v = warp_sum_d(acc[t]);
        if (lane == 0) red[wid][t] = v;
    }
    __syncthreads();
    if (threadIdx.x < kEnergyTerms) {
        double v = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) v += red[w][threadIdx.x];
        partial[blockIdx.x * kEnergyTerms + threadIdx.x] = v;
    }
}

int energy_blocks(int n) {
    const int b = blocks_for(n, kThreads);
    return b < kEnergyBlocks ? (b > 0 ? b : 1) : kEnergyBlocks;
}

void launch_energy(const Params &P, const DevBufs &B, int buf, const double g[3], double *partial, cudaStream_t s) {
    k_energy<<<energy_blocks(P.n), kThreads, 0, s>>>(P.n, B.pos[buf], B.vel[buf], (double)P.mass, g[0], g[1], g[2],
                                                     partial);
}

void launch_pseudo_viscosity(const Params &P, const DevBufs &B, int new_buf, float factor,
                             cudaStream_t s) {
    BBG_PBEGIN(B, KID_PSEUDO_VISCOSITY, s, -1);
    k_pv_aggregate<<<blocks_for(P.n, B.tune.block), B.tune.block, 0, s>>>(
        P, B.pos[1 - new_buf], B.pos[new_buf], B.vel[new_buf], B.inv_rho, B.cell, B.start, B.list, B.nbr,
        B.smoothed);
    k_pv_interpolate<<<blocks_for(P.n, kThreads), kThreads, 0, s>>>(P.n, B.vel[new_buf], B.smoothed,
                                                                    factor);
    BBG_PEND(B, s);
}

}  // namespace bbg
