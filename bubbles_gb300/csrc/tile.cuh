// tile.cuh -- tiles of the neighbour passes and the neighbour lists.
//
// The neighbour passes run one thread per particle in blocks of consecutive slots of the
// cell-sorted arrays (a "tile": the block size, 64 to 256, a tuning parameter), but for the fewest
// particles, which get several lanes each (sph.cu).
//
// The density pass records each particle's neighbour set (the reference bucket) as a
// list, member-major: entry q of particle i is list[q * n + i], so entry q of 32
// particles is written and read with one coalesced access.  Later passes request several
// entries and then the neighbours' records before using any (tile_members).  A particle
// with more than kMaxList members is "wide" (kWide in its cell word) and re-tests its 27
// cells exactly on every pass instead.
//
// Entries are absolute slot indices (32 bit).
#pragma once

#include <cuda_fp16.h>

#include "bbg_internal.cuh"

namespace bbg {

constexpr int kTile = 128;          // default tile: slots per tile = threads per block
constexpr int kMaxTile = 256;       // largest block size a neighbour pass is launched with
#ifndef BBG_GATHER_BATCH
#define BBG_GATHER_BATCH 4
#endif
// members whose neighbour records are requested together (build-time tuning knob)
constexpr int kGatherBatch = BBG_GATHER_BATCH;
using ListEntry = unsigned;

// Tile of block b among `tiles`.  With P.tile_sms = G > 0, blocks b, b + G, b + 2G, ... take
// consecutive tiles: tile = (b mod G) * per + b / G, per = ceil(tiles / G).  The block
// scheduler's first waves place those blocks on the same SM (one block per SM per round), so
// the blocks resident on an SM walk neighbouring tiles and share neighbour records in its L1.
// The grid is G * per blocks; a block whose tile is past the last one has no work.
__device__ __forceinline__ int tile_of_block(const Params &P, int b, int tiles) {
    const int G = P.tile_sms;
    if (G <= 0) return b;
    const int per = (tiles + G - 1) / G;
    return (b % G) * per + b / G;
}

// Where the density pass's filter sees a particle of cell (cx, cy, cz): its offset from the
// cell's lower corner in units of the longest cell side, or NaN when it does not lie in the cell
// (clamped into the grid, moved since the grid update), which the filter never drops.
__device__ __forceinline__ v3 filter_offset(const Params &P, float4 p, int cx, int cy, int cz) {
    const GridDev &g = P.g;
    const float x = (p.x - (g.minp[0] + (float)cx * g.len[0])) * P.filt_unit;
    const float y = (p.y - (g.minp[1] + (float)cy * g.len[1])) * P.filt_unit;
    const float z = (p.z - (g.minp[2] + (float)cz * g.len[2])) * P.filt_unit;
    const float lo = -P.filt_edge, hi = P.filt_edge;
    const bool in = x >= lo && x <= P.filt_side[0] + hi && y >= lo && y <= P.filt_side[1] + hi && z >= lo &&
                    z <= P.filt_side[2] + hi;
    const float nan = __int_as_float(0x7fffffff);
    return in ? V(x, y, z) : V(nan, nan, nan);
}

__device__ __forceinline__ void cell_coords(const GridDev &g, unsigned c, int &cx, int &cy, int &cz) {
    const unsigned plane = (unsigned)g.nx * (unsigned)g.ny;
    cz = (int)(c / plane);
    const unsigned rem = c - (unsigned)cz * plane;
    cy = (int)(rem / (unsigned)g.nx);
    cx = (int)(rem - (unsigned)cy * (unsigned)g.nx);
}

// Slot i of the density pass's filter: positions in half precision, slots 8k .. 8k + 7 in a record of
// four rows of eight halves, x, y, z and x'.  y and z are offsets from the centre of the
// particle's own cell; x counts cells modulo 4 from the middle of a window of four, x' with the
// window two cells on, so that the three cells around any cell lie in one of the two windows.
__device__ __forceinline__ void filter_record(const Params &P, float4 p, unsigned c, unsigned i, __half *rec) {
    int cx, cy, cz;
    cell_coords(P.g, c, cx, cy, cz);
    const v3 f = filter_offset(P, p, cx, cy, cz);
    __half *r = rec + 32 * (size_t)(i >> 3) + (i & 7u);
    r[0] = __float2half_rn((float)((cx & 3) - 2) * P.filt_side[0] + f.x);
    r[8] = __float2half_rn(f.y - 0.5f * P.filt_side[1]);
    r[16] = __float2half_rn(f.z - 0.5f * P.filt_side[2]);
    r[24] = __float2half_rn((float)(((cx + 2) & 3) - 2) * P.filt_side[0] + f.x);
}

// The 9 row ranges of the 27 neighbour cells of cell c in z, y, x order: f(r, b, e) for
// range r = slots [b, e).
template <class F>
__device__ __forceinline__ void tile_rows(const GridDev &g, const unsigned *__restrict__ start, unsigned c,
                                          F &&f) {
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const unsigned plane = (unsigned)nx * (unsigned)ny;
    const int cz = (int)(c / plane);
    const unsigned rem = c - (unsigned)cz * plane;
    const int cy = (int)(rem / (unsigned)nx);
    const int cx = (int)(rem - (unsigned)cy * (unsigned)nx);
    const int x0 = cx > 0 ? cx - 1 : 0;
    const int x1 = cx + 1 < nx ? cx + 1 : nx - 1;
    const int z0 = cz > 0 ? cz - 1 : 0, z1 = cz + 1 < nz ? cz + 1 : nz - 1;
    const int y0 = cy > 0 ? cy - 1 : 0, y1 = cy + 1 < ny ? cy + 1 : ny - 1;
    for (int z = z0; z <= z1; ++z) {
        for (int y = y0; y <= y1; ++y) {
            const unsigned row = (unsigned)y * (unsigned)nx + (unsigned)z * plane;
            f((z - cz + 1) * 3 + (y - cy + 1), __ldg(&start[row + (unsigned)x0]),
              __ldg(&start[row + (unsigned)x1 + 1u]));
        }
    }
}

// The 9 row ranges of the 27 neighbour cells of cell c (reference neighbour list,
// src/core/grid.h:555-593) in z, y, x order: f(j, r) for every candidate slot j of range r.
template <class F>
__device__ __forceinline__ void tile_candidates(const GridDev &g, const unsigned *__restrict__ start,
                                                unsigned c, F &&f) {
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const unsigned plane = (unsigned)nx * (unsigned)ny;
    const int cz = (int)(c / plane);
    const unsigned rem = c - (unsigned)cz * plane;
    const int cy = (int)(rem / (unsigned)nx);
    const int cx = (int)(rem - (unsigned)cy * (unsigned)nx);
    const int x0 = cx > 0 ? cx - 1 : 0;
    const int x1 = cx + 1 < nx ? cx + 1 : nx - 1;
    const int z0 = cz > 0 ? cz - 1 : 0, z1 = cz + 1 < nz ? cz + 1 : nz - 1;
    const int y0 = cy > 0 ? cy - 1 : 0, y1 = cy + 1 < ny ? cy + 1 : ny - 1;
    for (int z = z0; z <= z1; ++z) {
        for (int y = y0; y <= y1; ++y) {
            const int r = (z - cz + 1) * 3 + (y - cy + 1);
            const unsigned row = (unsigned)y * (unsigned)nx + (unsigned)z * plane;
            const unsigned b = __ldg(&start[row + (unsigned)x0]);
            const unsigned e = __ldg(&start[row + (unsigned)x1 + 1u]);
            for (unsigned j = b; j < e; ++j) f(j, r);
        }
    }
}

// Number of candidates in the 27 cells of cell c.
__device__ __forceinline__ unsigned candidate_count(const GridDev &g, const unsigned *__restrict__ start,
                                                    unsigned c) {
    unsigned total = 0;
    tile_rows(g, start, c, [&](int, unsigned b, unsigned e) { total += e - b; });
    return total;
}

// For every member j != i of particle i's step-start neighbour set: use(fetch(j)).
// Members are processed NB at a time: the NB list entries and then the NB neighbour
// records are requested before any is used (entries past the end fetch particle i
// itself and are not used).  Wide particles re-test their candidates with the
// exact membership test at the step-start positions pos0.
template <int NB = kGatherBatch, bool SPLIT = false, class Fetch, class Use>
__device__ __forceinline__ void tile_members(const Params &P, const unsigned *__restrict__ start,
                                             const ListEntry *__restrict__ list,
                                             const int *__restrict__ nbr, const float4 *__restrict__ pos0,
                                             unsigned cellw, int i, Fetch &&fetch, Use &&use) {
    if (cellw & kWide) {
        if (candidate_count(P.g, start, cellw & ~kWide) > kMaxCandidates) return;
        const float4 pi = __ldg(&pos0[i]);
        tile_candidates(P.g, start, cellw & ~kWide, [&](unsigned j, int) {
            if (j == (unsigned)i) return;
            const float4 pj = __ldg(&pos0[j]);
            if (std_member(P, pi, pj, dist2(pi, pj))) use(fetch(j));
        });
        return;
    }
    const int cnt = __ldg(&nbr[i]) - 1;   // members other than i
    const size_t n = (size_t)P.n;
    const ListEntry *l = list + i;        // entry q + k of the group at l + k * n
    // SPLIT: whole groups without per-member predicates, then the partial group (a second
    // copy of `use`: measured faster for the small predicted-density body only)
    const int full = SPLIT ? cnt - cnt % NB : 0;
    int q = 0;
    for (; q < full; q += NB, l += NB * n) {
        unsigned j[NB];
#pragma unroll
        for (int k = 0; k < NB; k++) j[k] = __ldg(l + k * n);
        decltype(fetch(0u)) d[NB];
#pragma unroll
        for (int k = 0; k < NB; k++) d[k] = fetch(j[k]);
#pragma unroll
        for (int k = 0; k < NB; k++) use(d[k]);
    }
    for (; q < cnt; q += NB, l += NB * n) {   // predicated groups (with SPLIT: the last one)
        unsigned j[NB];
#pragma unroll
        for (int k = 0; k < NB; k++) j[k] = q + k < cnt ? __ldg(l + k * n) : (unsigned)i;
        decltype(fetch(0u)) d[NB];
#pragma unroll
        for (int k = 0; k < NB; k++) d[k] = fetch(j[k]);
#pragma unroll
        for (int k = 0; k < NB; k++)
            if (q + k < cnt) use(d[k]);
    }
}

}  // namespace bbg
