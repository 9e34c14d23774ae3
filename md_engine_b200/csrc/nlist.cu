// Cell-binned neighbour list (the GridGPU component, src/GridGPU.cu:824-1103).
//
// Differences from the reference's launch structure (the pair SET is the
// same, see below):
//  * no host round trips: the rebuild decision (setBuildFlag, GridGPU.cu:755),
//    the cell histogram, the exclusive scan (host cumulativeSum at
//    GridGPU.cu:902-908) and the list sizing all stay on the device; every
//    kernel of the rebuild group reads DeviceStatus::rebuild and returns
//    immediately when no rebuild is due, so the group can sit inside a
//    captured CUDA graph.
//  * search cells are >= cut/m wide (m <= 4: a (2m+1)^3 stencil walked as
//    (2m+1)^2 contiguous z-rows) instead of >= cut with 27 cells; the atoms tested are
//    a superset of every pair within cut, and each pair is tested once with
//    the minimum-image shift, so the pair set is unchanged.
//  * atoms are ordered by (cell, type, id) -- deterministic -- instead of the
//    atomicAdd arrival order of countNumInGridCells (GridGPU.cu:190-203).
//  * one sweep writes the list into a fixed per-atom capacity (overflow is
//    flagged in the status word) instead of count + max + prefix + assign.
//
// The predicate is the reference's FP32 expression (GridGPU.cu:326-338,
// 518-522): d = (x_j + shift) - x_i, r2 = dot(d, d) as nvcc contracts it,
// fma(dz, dz, fma(dy, dy, dx*dx)), pair kept iff r2 < cut*cut (float).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "engine.hpp"

namespace mdx {

namespace {

__device__ __forceinline__ int cell_coord(float x, float lo, float inv_ds, int n) {
    int c = (int)((x - lo) * inv_ds);
    return c < 0 ? 0 : (c >= n ? n - 1 : c);
}

struct CellGrid {
    float3 lo;
    float3 inv_ds;
    int3 ns;
};

__device__ __forceinline__ int cell_of_pos(const CellGrid &g, float3 p) {
    int cx = cell_coord(p.x, g.lo.x, g.inv_ds.x, g.ns.x);
    int cy = cell_coord(p.y, g.lo.y, g.inv_ds.y, g.ns.y);
    int cz = cell_coord(p.z, g.lo.z, g.inv_ds.z, g.ns.z);
    return (cx * g.ns.y + cy) * g.ns.z + cz;
}

// Arguments of the rebuild-group kernels for one system.  Every kernel takes
// a0 (single system) and tab (batched replicas: tab[blockIdx.y], a0 is then
// only the largest replica used to size the grid).
struct GridArgs {
    float4 *xs, *vs, *fs;
    float *qs;
    uint32_t *ids;
    float4 *xs2, *vs2, *fs2;
    float *qs2;
    uint32_t *ids2;
    float4 *xs_last;
    int *idToIdx;
    int *cell_of;
    uint32_t *cell_count, *cell_start, *cell_fill;
    int *perm_tmp;
    DeviceStatus *st;
    Box box;
    CellGrid g;
    int n, ncell, interval;
    float skin2q;
    // 1: a list build into the alternate buffers only (the molecule form's
    // per-site list for Grid.getNeighborList): idToIdx, the primary streams
    // and the build counter are left alone
    int view;
};
#define MDX_GRID_ARGS \
    pdl_wait();       \
    const GridArgs A = tab ? tab[blockIdx.y] : a0

// setBuildFlag (GridGPU.cu:755-774) + the periodicInterval gate of
// IntegratorVerlet.cu:696: rebuild iff forced, or turn % interval == 0 and
// any atom moved more than skin/2 since the last build.
__global__ void k_check(const GridArgs a0, const GridArgs *__restrict__ tab, int force) {
    MDX_GRID_ARGS;
    DeviceStatus *st = A.st;
    if (!force) {
        long long t = st->turn;
        if (A.interval <= 0 || (t % A.interval) != 0) return;
    } else {
        if (blockIdx.x == 0 && threadIdx.x == 0) st->rebuild = 1u;
        return;
    }
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int moved = 0;
    if (i < A.n) {
        float3 d = min_image(A.box, f3(A.xs[i]) - f3(A.xs_last[i]));
        moved = dot3(d, d) > A.skin2q;
    }
    if (__syncthreads_or(moved) && threadIdx.x == 0) atomicOr(&st->rebuild, 1u);
}

// periodicWrap (GridGPU.cu:138-161) + countNumInGridCells (GridGPU.cu:190-203)
__global__ void k_wrap_bin(const GridArgs a0, const GridArgs *__restrict__ tab) {
    MDX_GRID_ARGS;
    if (!A.st->rebuild) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    const Box &box = A.box;
    float4 p = A.xs[i];
    float ix = floorf((p.x - box.lo.x) / box.L.x);
    float iy = floorf((p.y - box.lo.y) / box.L.y);
    float iz = floorf((p.z - box.lo.z) / box.L.z);
    if (ix != 0.f || iy != 0.f || iz != 0.f) {
        p.x = p.x - box.L.x * ix;
        p.y = p.y - box.L.y * iy;
        p.z = p.z - box.L.z * iz;
        if (!A.view) A.xs[i] = p;  // a view build wraps its sorted copy only (k_gather)
    }
    int c = cell_of_pos(A.g, f3(p));
    A.cell_of[i] = c;
    atomicAdd(A.cell_count + c, 1u);
}

// exclusive scan of the cell histogram (replaces the host cumulativeSum,
// helpers.h:15-24); also clears the fill counters.  Tiles of kScanTile cells,
// a block for each up to kScanBlocks, beyond that a block for as many in a
// row as share them out: it sums the counts before its tiles itself (coalesced
// 16-byte loads from L2, no block waits for another), then scans them one
// after another -- through shared memory, thread t its eight consecutive cells
// in registers, warp and block totals by shuffles.  One block walking all
// tiles took 5.6 us a tile: 74 us for the 104,000 cells of 256,000 particles,
// 6 us so.  With a block to every tile, whatever their number, the counts read
// again grow with the square of the cells: rebuild of 4,000 atoms in a dilute
// box of 20 million cells 8.6 ms, 5.5 so (20.7 with one block); of 4 million
// 1.01, 0.93.
constexpr int kScanThreads = 1024;
constexpr int kScanPer = 8;
constexpr int kScanTile = kScanThreads * kScanPer;
constexpr int kScanBlocks = 128;
__host__ __device__ inline int scan_tiles(int ncell) { return (ncell + kScanTile - 1) / kScanTile; }
inline unsigned scan_blocks(int ncell) { return (unsigned)std::min(scan_tiles(ncell), kScanBlocks); }
__global__ void __launch_bounds__(kScanThreads) k_scan_cells(const GridArgs a0, const GridArgs *__restrict__ tab) {
    MDX_GRID_ARGS;
    if (!A.st->rebuild) return;
    const uint32_t *__restrict__ count = A.cell_count;
    const int ncell = A.ncell;
    const int mine = (scan_tiles(ncell) + kScanBlocks - 1) / kScanBlocks * kScanTile;  // a block's cells
    if ((long long)blockIdx.x * mine >= ncell) return;
    const int first = (int)blockIdx.x * mine, end = first + min(mine, ncell - first);
    __shared__ uint4 tile4[kScanTile / 4];
    __shared__ uint32_t warp_tot[32], warp_before[32];
    uint32_t *const tile = reinterpret_cast<uint32_t *>(tile4);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t before = 0u;  // this thread's share of the counts before the tile
    {
        const uint4 *c4 = reinterpret_cast<const uint4 *>(count);
#pragma unroll 4
        for (int k = threadIdx.x; k < first / 4; k += kScanThreads) {
            const uint4 c = c4[k];
            before += c.x + c.y + c.z + c.w;
        }
    }
#pragma unroll 1
    for (int base = first;;) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
        if (lane == 0) warp_before[w] = before;
        const int nt = min(kScanTile, end - base);
#pragma unroll
        for (int k = 0; k < kScanPer; k++) {
            const int c = k * kScanThreads + (int)threadIdx.x;
            tile[c] = c < nt ? count[base + c] : 0u;
        }
        __syncthreads();
        const uint4 a = tile4[2 * threadIdx.x], b = tile4[2 * threadIdx.x + 1];
        const uint32_t v[kScanPer] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t run = 0u;
#pragma unroll
        for (int k = 0; k < kScanPer; k++) run += v[k];
        uint32_t x = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[w] = x;
        __syncthreads();
        if (w == 0) {
            uint32_t t = warp_tot[lane], bf = warp_before[lane];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) bf += __shfl_xor_sync(0xffffffffu, bf, o);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += y;
            }
            warp_tot[lane] = bf + t;  // everything up to and with the warp
        }
        __syncthreads();
        const uint32_t last = warp_tot[w];
        uint32_t excl = last - __shfl_sync(0xffffffffu, x, 31) + x - run;
        uint32_t e[kScanPer];
#pragma unroll
        for (int k = 0; k < kScanPer; k++) {
            e[k] = excl;
            excl += v[k];
        }
        tile4[2 * threadIdx.x] = make_uint4(e[0], e[1], e[2], e[3]);
        tile4[2 * threadIdx.x + 1] = make_uint4(e[4], e[5], e[6], e[7]);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kScanPer; k++) {
            const int c = k * kScanThreads + (int)threadIdx.x;
            if (c < nt) {
                A.cell_start[base + c] = tile[c];
                A.cell_fill[base + c] = 0u;
            }
        }
        if (base + nt == ncell && threadIdx.x == kScanThreads - 1) A.cell_start[ncell] = excl;
        base += nt;
        if (base >= end) break;
        before = threadIdx.x == 0 ? warp_tot[31] : 0u;  // everything up to the tile's end
        __syncthreads();  // the tile and the totals are written again
    }
}

__global__ void k_scatter(const GridArgs a0, const GridArgs *__restrict__ tab) {
    MDX_GRID_ARGS;
    if (!A.st->rebuild) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    int c = A.cell_of[i];
    uint32_t slot = atomicAdd(A.cell_fill + c, 1u);
    A.perm_tmp[A.cell_start[c] + slot] = i;
}

// sortPerAtomArrays (GridGPU.cu:253-293): each atom's place in its cell, the
// rank of (type, id) among the cell's few atoms (deterministic order), then
// every stream into the alternate buffers and idToIdx rebuilt.  One thread per
// atom (a warp per cell had most lanes idle at two atoms a cell: 28 us and a
// launch of its own at 256,000 atoms).  The histogram is cleared for the next
// build.
__global__ void k_gather(const GridArgs a0, const GridArgs *__restrict__ tab) {
    MDX_GRID_ARGS;
    if (!A.st->rebuild) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    for (int c = p; c < A.ncell; c += gridDim.x * blockDim.x) A.cell_count[c] = 0u;
    if (p >= A.n) return;
    const int s = A.perm_tmp[p];
    const int c = A.cell_of[s];
    const uint32_t beg = A.cell_start[c], end = A.cell_start[c + 1];
    float4 x = A.xs[s];
    const uint32_t id = A.ids[s];
    const unsigned long long ka = ((unsigned long long)(uint32_t)type_of(x) << 32) | id;
    uint32_t d = beg;
    for (uint32_t q = beg; q < end; q++) {
        const int b = A.perm_tmp[q];
        const unsigned long long kb = ((unsigned long long)(uint32_t)type_of(A.xs[b]) << 32) | A.ids[b];
        d += kb < ka;
    }
    if (A.view) {
        // the view build's copy, wrapped as k_wrap_bin wraps in place
        const Box &box = A.box;
        const float ix = floorf((x.x - box.lo.x) / box.L.x);
        const float iy = floorf((x.y - box.lo.y) / box.L.y);
        const float iz = floorf((x.z - box.lo.z) / box.L.z);
        if (ix != 0.f || iy != 0.f || iz != 0.f) {
            x.x = x.x - box.L.x * ix;
            x.y = x.y - box.L.y * iy;
            x.z = x.z - box.L.z * iz;
        }
    }
    A.xs2[d] = x;
    A.vs2[d] = A.vs[s];
    A.fs2[d] = A.fs[s];
    A.qs2[d] = A.qs[s];
    A.ids2[d] = id;
    if (!A.view) A.idToIdx[id] = d;
}

// the sorted streams back into the primary buffers (the captured graph keeps
// the same pointers), and the positions of this list build for the skin check
__global__ void k_copyback(const GridArgs a0, const GridArgs *__restrict__ tab) {
    MDX_GRID_ARGS;
    if (!A.st->rebuild) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    const float4 p = A.xs2[i];
    A.xs[i] = p;
    A.xs_last[i] = p;
    A.vs[i] = A.vs2[i];
    A.fs[i] = A.fs2[i];
    A.qs[i] = A.qs2[i];
    A.ids[i] = A.ids2[i];
}

// assignNeighbors / assignFromCell (GridGPU.cu:482-734) with the exclusion
// lookup of addExclusion (GridGPU.cu:466-478), one warp per home cell.
// The candidates of the cell -- its (2m+1)^2 stencil rows, each row's z range
// and each row trimmed to the cells that can hold a point within cut of the
// home atoms' bounding box (conservative margin of 1e-3 cell) -- are laid out
// as one sequence of contiguous segments of the sorted streams.  The warp
// walks that sequence 32 candidates at a time, one candidate per lane,
// already shifted by its periodic image (x_j + shift, the reference's first
// rounding), for HG home atoms at once held in registers.  The sequence is
// first expanded into shared memory (sorted index and image code per
// candidate, windows of kCandWin) so a chunk costs one shared load; every lane tests
// its candidate against each of them with the reference's predicate and two
// ballots give the hit and the "can interact" masks.  The warp owns whole
// rows, so a single pass writes them: interacting pairs at the front,
// provably zero ones at the back, each slot from the running counts (the same
// in every lane) plus a popcount of the lower lanes' hits -- deterministic,
// and the entries written for one home atom at a time are consecutive slots
// of its row.  Exclusion depths come from the id-window bit planes (the id
// list only for atoms with far exclusions).  COUNT counts alone to size the
// first build.
constexpr int kBuildCellsPerBlock = 4;            // one warp per cell
constexpr int kStencilMax = 4;                    // largest m (cells >= cut/m)
constexpr int kBuildSegMax = 2 * (2 * kStencilMax + 1) * (2 * kStencilMax + 1);  // two z segments per row
constexpr int kCandWin = 1536;                    // expanded candidates per warp and window
constexpr int kCandIdxBits = 27;                  // sorted index bits of an expanded candidate
constexpr int kCandPad = 64;                      // harmless entries after a window (branch-free prefetch)
constexpr uint32_t kNoShift = 13u;                // image code (1,1,1): no shift

struct BuildArgs {
    const float4 *xs2, *vs2, *fs2;
    const float *qs2;
    const uint32_t *ids2;
    float4 *xs, *vs, *fs;
    float *qs;
    uint32_t *ids;
    float4 *xs_last;
    const uint32_t *cell_start;
    const int *excl_start;
    const uint32_t *excl_ids;
    const ulonglong2 *excl_win;
    const uint8_t *excl_far;
    const uint32_t *ljmask;
    uint32_t *counts, *counts_int, *nlist;
    DeviceStatus *st;
    CellGrid g;
    Box box;
    int ncell, m, use_excl, part_q, cap;
    int parts;  // warps per cell
    float cutsq;
};

// exclusion depth of the pair (home id myid, candidate id oid): bit planes of
// the id window (w, in registers), else the id list of an atom with far
// exclusions
__device__ __forceinline__ uint32_t excl_depth(const BuildArgs &A, uint32_t myid, bool far, ulonglong2 w,
                                               uint32_t oid) {
    const uint32_t dd = oid - myid + 32u;
    uint32_t depth = 0u;
    if (dd < 64u) depth = (uint32_t)((w.x >> dd) & 1ull) | ((uint32_t)((w.y >> dd) & 1ull) << 1);
    if (far && depth == 0u) {
        for (int e = A.excl_start[myid]; e < A.excl_start[myid + 1]; e++) {
            const uint32_t x = A.excl_ids[e];
            if ((x & kExclMask) == oid) {
                depth = x >> 30;
                break;
            }
        }
    }
    return depth;
}

// SPLIT: interacting pairs to the front of a row, provably zero ones to the
// back (ljmask, part_q); EXCL: exclusion depths from the id window.  Both are
// compile-time so that the candidate loop carries no tests for them.
// STRIDE 4: the molecule-pair list of the molecule form (molecules by the
// position of their site 0, at 4 k; neither split nor exclusions).
template <int TP, int HG, bool COUNT, bool SPLIT, bool EXCL, int STRIDE = 1>
__global__ void __launch_bounds__(kBuildCellsPerBlock * 32, 7) k_build_cells(const BuildArgs a0,
                                                                            const BuildArgs *__restrict__ tab) {
    pdl_wait();
    const BuildArgs A = tab ? tab[blockIdx.y] : a0;
    if (!COUNT && !A.st->rebuild) return;
    constexpr int GP = 32 / TP;
    // segment table: offset in the sequence | image code << kCandIdxBits,
    // and the first sorted index (two words per segment: seven blocks fit
    // an SM beside the candidate windows)
    __shared__ uint32_t sh_seg_offc_all[kBuildCellsPerBlock][kBuildSegMax + 1];
    __shared__ int sh_seg_beg_all[kBuildCellsPerBlock][kBuildSegMax];
    __shared__ uint32_t sh_cand_all[kBuildCellsPerBlock][kCandWin + kCandPad];
    __shared__ float4 sh_shift[27];  // image shift by code (ix+1) + 3 (iy+1) + 9 (iz+1)
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    if (threadIdx.x < 27) {
        const int t = threadIdx.x;
        sh_shift[t] = make_float4((float)(t % 3 - 1) * A.box.L.x, (float)(t / 3 % 3 - 1) * A.box.L.y,
                                  (float)(t / 9 - 1) * A.box.L.z, 0.f);
    }
    __syncthreads();  // the only block-wide barrier: warps own cells from here on
    // parts warps share a cell's home groups of HG in turn
    const int parts = A.parts, gw = blockIdx.x * kBuildCellsPerBlock + wib;
    const int c = gw / parts, part = gw - c * parts;
    if (c >= A.ncell) return;
    uint32_t *const sh_seg_offc = sh_seg_offc_all[wib];
    int *const sh_seg_beg = sh_seg_beg_all[wib];
    uint32_t *const sh_cand = sh_cand_all[wib];
    const CellGrid &g = A.g;
    const int cs = (int)A.cell_start[c], ce = (int)A.cell_start[c + 1];
    if (ce <= cs + HG * part) return;
    const int cz = c % g.ns.z, cy = (c / g.ns.z) % g.ns.y, cx = c / (g.ns.z * g.ns.y);
    const int m = A.m, side = 2 * m + 1;
    const float cutsq = A.cutsq;
    const uint32_t cap = (uint32_t)A.cap;
    uint32_t *const nlist = A.nlist;
    const float dsx = 1.0f / g.inv_ds.x, dsy = 1.0f / g.inv_ds.y, dsz = 1.0f / g.inv_ds.z;
    const uint32_t lt = (1u << lane) - 1u;
    // bounding box of this warp's home atoms
    float bxl = 3.0e38f, bxh = -3.0e38f, byl = 3.0e38f, byh = -3.0e38f, bzl = 3.0e38f, bzh = -3.0e38f;
    for (int i = cs + lane; i < ce; i += 32) {
        if (parts > 1 && (i - cs) / HG % parts != part) continue;
        const float4 p4 = A.xs2[STRIDE * i];
        bxl = fminf(bxl, p4.x);
        bxh = fmaxf(bxh, p4.x);
        byl = fminf(byl, p4.y);
        byh = fmaxf(byh, p4.y);
        bzl = fminf(bzl, p4.z);
        bzh = fmaxf(bzh, p4.z);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        bxl = fminf(bxl, __shfl_xor_sync(0xffffffffu, bxl, o));
        bxh = fmaxf(bxh, __shfl_xor_sync(0xffffffffu, bxh, o));
        byl = fminf(byl, __shfl_xor_sync(0xffffffffu, byl, o));
        byh = fmaxf(byh, __shfl_xor_sync(0xffffffffu, byh, o));
        bzl = fminf(bzl, __shfl_xor_sync(0xffffffffu, bzl, o));
        bzh = fmaxf(bzh, __shfl_xor_sync(0xffffffffu, bzh, o));
    }
    // segment table: lane r builds stencil row r's z segments, rows in
    // chunks of 32 with the running totals carried
    int seg_base = 0, cand_base = 0;
    for (int r0 = 0; r0 < side * side; r0 += 32) {
        // up to two segments per row (the stencil wraps at most once):
        // the parts of the z range below, inside and above the box
        int nseg = 0, b0 = 0, l0 = 0, b1 = 0, l1 = 0;
        uint32_t cxy = 0u, cz0 = 0u, cz1 = 0u;  // image codes
        const int r = r0 + lane;
        if (r < side * side) {
            const int kx = cx - m + r / side, ky = cy - m + r % side;
            const int kxw = kx < 0 ? kx + g.ns.x : (kx >= g.ns.x ? kx - g.ns.x : kx);
            const uint32_t ix = kx < 0 ? 0u : (kx >= g.ns.x ? 2u : 1u);
            const int kyw = ky < 0 ? ky + g.ns.y : (ky >= g.ns.y ? ky - g.ns.y : ky);
            const uint32_t iy = ky < 0 ? 0u : (ky >= g.ns.y ? 2u : 1u);
            cxy = ix + 3u * iy;
            // distance from the home box to this row of cells (image
            // frame), shrunk by the margin
            const float clx = g.lo.x + (float)kx * dsx;
            const float cly = g.lo.y + (float)ky * dsy;
            float dxm = fmaxf(fmaxf(clx - bxh, bxl - (clx + dsx)), 0.f);
            float dym = fmaxf(fmaxf(cly - byh, byl - (cly + dsy)), 0.f);
            dxm = fmaxf(dxm - 1e-3f * dsx, 0.f);
            dym = fmaxf(dym - 1e-3f * dsy, 0.f);
            const float rz2 = cutsq - dxm * dxm - dym * dym;
            if (rz2 > 0.f) {
                const float rz = sqrtf(rz2) + 1e-3f * dsz;
                const int zlo = max(cz - m, (int)floorf((bzl - rz - g.lo.z) * g.inv_ds.z));
                const int zhi = min(cz + m, (int)floorf((bzh + rz - g.lo.z) * g.inv_ds.z));
                const int rowbase = (kxw * g.ns.y + kyw) * g.ns.z;
#pragma unroll
                for (int part = 0; part < 3; part++) {
                    const int za = part == 0 ? zlo : (part == 1 ? max(zlo, 0) : max(zlo, g.ns.z));
                    const int ze = part == 0 ? min(zhi, -1) : (part == 1 ? min(zhi, g.ns.z - 1) : zhi);
                    const int wrap = part == 0 ? g.ns.z : (part == 1 ? 0 : -g.ns.z);
                    const uint32_t czp = 9u * (uint32_t)part;
                    if (za <= ze) {
                        const int pbeg = (int)A.cell_start[rowbase + za + wrap];
                        const int pend = (int)A.cell_start[rowbase + ze + wrap + 1];
                        if (pend > pbeg) {
                            if (nseg == 0) {
                                b0 = pbeg;
                                l0 = pend - pbeg;
                                cz0 = czp;
                            } else {
                                b1 = pbeg;
                                l1 = pend - pbeg;
                                cz1 = czp;
                            }
                            nseg++;
                        }
                    }
                }
            }
        }
        // inclusive scans of the segment counts and lengths
        int so = nseg, lo = l0 + l1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, so, o);
            const int b = __shfl_up_sync(0xffffffffu, lo, o);
            if (lane >= o) {
                so += a;
                lo += b;
            }
        }
        const int slot = seg_base + so - nseg, off = cand_base + lo - (l0 + l1);
        if (nseg > 0) {
            sh_seg_beg[slot] = b0;
            sh_seg_offc[slot] = (uint32_t)off | ((cxy + cz0) << kCandIdxBits);
        }
        if (nseg > 1) {
            sh_seg_beg[slot + 1] = b1;
            sh_seg_offc[slot + 1] = (uint32_t)(off + l0) | ((cxy + cz1) << kCandIdxBits);
        }
        // the first window straight from the rows, every lane its own
        // segments (later windows of a long sequence expand from the table)
        {
            const uint32_t w0c = (cxy + cz0) << kCandIdxBits, w1c = (cxy + cz1) << kCandIdxBits;
            const int e0 = min(off + l0, kCandWin), e1 = min(off + l0 + l1, kCandWin);
            for (int t = off; t < e0; t++) sh_cand[t] = (uint32_t)(b0 - off + t) | w0c;
            for (int t = off + l0; t < e1; t++) sh_cand[t] = (uint32_t)(b1 - off - l0 + t) | w1c;
        }
        seg_base += __shfl_sync(0xffffffffu, so, 31);
        cand_base += __shfl_sync(0xffffffffu, lo, 31);
    }
    if (lane == 0) sh_seg_offc[seg_base] = (uint32_t)cand_base;  // total candidates

    __syncwarp();
    const int nseg = seg_base;
    const int total = cand_base;
    if (total >= (1 << kCandIdxBits)) {  // the packed table offset cannot hold it
        if (lane == 0) atomicOr(&A.st->bits, kStatusNlistOverflow);
        return;
    }

    // the prefetch reads up to kCandPad entries past a window: the cell's
    // first site, unshifted (in bounds, never counted)
    auto pad = [&](int wn) {
        for (int t = wn + lane; t < wn + kCandPad; t += 32) sh_cand[t] = (uint32_t)cs | (kNoShift << kCandIdxBits);
    };
    // expand candidates [w0, w0 + wn) of the segment sequence into sh_cand
    auto expand = [&](int w0, int wn) {
        __syncwarp();
        for (int sg = 0; sg < nseg; sg++) {
            constexpr uint32_t kOffMask = (1u << kCandIdxBits) - 1u;
            const uint32_t oc = sh_seg_offc[sg];
            const int off = (int)(oc & kOffMask);
            const int lo = max(off, w0), hi = min((int)(sh_seg_offc[sg + 1] & kOffMask), w0 + wn);
            const uint32_t beg = (uint32_t)(sh_seg_beg[sg] - off), code = oc & ~kOffMask;
            for (int t = lo + lane; t < hi; t += 32) sh_cand[t - w0] = (beg + (uint32_t)t) | code;
        }
        pad(wn);
        __syncwarp();
    };
    const bool single = total <= kCandWin;
    if (single) {
        pad(total);
        __syncwarp();
    }
    // home atoms HG at a time, in registers (warp-uniform values)
    for (int g0 = cs + HG * part; g0 < ce; g0 += HG * parts) {
        float hx[HG], hy[HG], hz[HG], hq[HG];
        uint32_t hmask[HG], hid[HG], ci[HG], cn[HG];
        ulonglong2 hwin[HG];
        bool hfar[HG];
        uint32_t *hrow[HG];
#pragma unroll
        for (int k = 0; k < HG; k++) {
            const int i = g0 + k;
            const bool v = i < ce;
            const int ii = v ? i : cs;
            const float4 p4 = A.xs2[STRIDE * ii];
            // an absent home slot sits far outside the box: r^2 overflows to
            // infinity and it never hits
            hx[k] = v ? p4.x : 3.0e37f;
            hy[k] = v ? p4.y : 3.0e37f;
            hz[k] = v ? p4.z : 3.0e37f;
            hq[k] = SPLIT && A.part_q ? A.qs2[ii] : 0.f;
            hmask[k] = SPLIT ? A.ljmask[type_of(p4)] : 0xffffffffu;
            hid[k] = EXCL ? A.ids2[ii] : 0u;
            hfar[k] = EXCL ? A.excl_far[hid[k]] != 0 : false;
            hwin[k] = EXCL ? A.excl_win[hid[k]] : make_ulonglong2(0ull, 0ull);
            hrow[k] = nlist + (size_t)(ii / GP) * cap * GP + (ii % GP) * TP;
            ci[k] = 0u;
            cn[k] = 0u;
        }
        for (int w0 = 0; w0 < total; w0 += kCandWin) {
            const int wn = min(kCandWin, total - w0);
            if (!single) expand(w0, wn);
            // candidate: sorted index, raw position, image shift, charge, id;
            // the next chunk's loads are issued before the current one is
            // tested (indices up to wn + 63 < wn + kCandPad: no bounds test)
            uint32_t pn = 0u, idn = 0u;
            float4 pjn, shn;
            float qn = 0.f;
            auto fetch = [&](int k) {
                const uint32_t e = sh_cand[k];
                pn = e & ((1u << kCandIdxBits) - 1u);
                shn = sh_shift[e >> kCandIdxBits];
                pjn = A.xs2[STRIDE * pn];
                if (SPLIT) qn = A.qs2[pn];
                if (EXCL) idn = A.ids2[pn];
            };
            fetch(lane);
#pragma unroll 2
            for (int c0 = 0; c0 < wn; c0 += 32) {
                const uint32_t p = pn;
                const bool cval = c0 + lane < wn;
                const float cxj = __fadd_rn(pjn.x, shn.x);
                const float cyj = __fadd_rn(pjn.y, shn.y);
                const float czj = __fadd_rn(pjn.z, shn.z);
                const uint32_t tj = (uint32_t)type_of(pjn);
                const float qj = qn;
                const uint32_t oid = idn;
                fetch(c0 + 32 + lane);
                bool hit[HG], act[HG];
                uint32_t hm[HG], am[HG];
#pragma unroll
                for (int k = 0; k < HG; k++) {
                    const float ddx = __fsub_rn(cxj, hx[k]);
                    const float ddy = __fsub_rn(cyj, hy[k]);
                    const float ddz = __fsub_rn(czj, hz[k]);
                    const float r2 = __fmaf_rn(ddz, ddz, __fmaf_rn(ddy, ddy, __fmul_rn(ddx, ddx)));
                    hit[k] = cval && r2 < cutsq && p != (uint32_t)(g0 + k);
                    hm[k] = __ballot_sync(0xffffffffu, hit[k]);
                    act[k] = true;
                    am[k] = hm[k];
                    if (SPLIT && !COUNT) {
                        act[k] = ((hmask[k] >> tj) & 1u) != 0u || hq[k] * qj != 0.f;
                        am[k] = __ballot_sync(0xffffffffu, hit[k] && act[k]);
                    }
                }
#pragma unroll
                for (int k = 0; k < HG; k++) {
                    if (COUNT) {
                        ci[k] += __popc(hm[k]);
                        continue;
                    }
                    if (hm[k] == 0u) continue;  // warp-uniform: no hit for this home in the chunk
                    const uint32_t before = __popc(hm[k] & lt);
                    const uint32_t bi = __popc(am[k] & lt);
                    const uint32_t pos = act[k] ? ci[k] + bi : cap - 1u - cn[k] - (before - bi);
                    uint32_t entry = p;
                    // a depth needs an id within 32 of the home's (the bit
                    // window) or a home with far exclusions; most chunks have
                    // neither
                    if (EXCL && (hfar[k] || __any_sync(0xffffffffu, hit[k] && oid - hid[k] + 32u < 64u)))
                        entry |= excl_depth(A, hid[k], hfar[k], hwin[k], oid) << 30;
                    if (hit[k] && ci[k] + cn[k] + before < cap) hrow[k][(pos / TP) * 32u + pos % TP] = entry;
                    const uint32_t na = __popc(am[k]);
                    ci[k] += na;
                    cn[k] += __popc(hm[k]) - na;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < HG; k++) {
            if (lane == k && g0 + k < ce) {
                const int i = g0 + k;
                const uint32_t cnt = ci[k] + cn[k];
                if (COUNT) {
                    atomicMax(&A.st->max_neighbors, cnt);
                } else {
                    A.counts[i] = cnt;
                    if (STRIDE == 1) A.counts_int[i] = ci[k];
                    if (cnt > cap) atomicOr(&A.st->bits, kStatusNlistOverflow);
                    atomicMax(STRIDE == 1 ? &A.st->max_neighbors : &A.st->max_mol_neighbors, cnt);
                }
            }
        }
    }
}

// the rebuild is over (one thread; the histogram was cleared by the sort)
__global__ void k_finish(const GridArgs a0, const GridArgs *__restrict__ tab) {
    MDX_GRID_ARGS;
    DeviceStatus *st = A.st;
    if (!st->rebuild) return;
    if (!A.view) st->n_builds += 1;
    st->rebuild = 0u;
}

// ---- molecule form (all-rigid four-site water) ---------------------------
// The sort unit is the molecule: its cell is the cell of its site 0, slots
// are ordered by (cell, molecule index), and slot d's sites land at 4d .. 4d+3
// of every per-atom stream.
struct MolGridArgs {
    float4 *xs, *vs, *fs;
    float *qs;
    uint32_t *ids;
    float4 *xs2, *vs2, *fs2;
    float *qs2;
    uint32_t *ids2;
    float4 *xs_last;
    int *idToIdx;
    int4 *mol_idx;      // FixRigid's molecule -> atom indices (rewritten by the sort)
    int4 *mol_idx_e3b;  // FixE3B's copy of the same molecules (may be null)
    int *cell_of;
    uint32_t *cell_count, *cell_start, *cell_fill;
    int *perm_tmp, *perm;
    DeviceStatus *st;
    Box box;
    CellGrid g;
    int nmol, ncell;
};

// one system (m0) or, for batched replicas, tab[blockIdx.y] (m0 then only
// sizes the grid; blocks past a smaller replica's work return at once)
#define MDX_MG_ARGS \
    pdl_wait();     \
    const MolGridArgs M = tab ? tab[blockIdx.y] : m0

__device__ __forceinline__ float4 wrap_pos(const Box &box, float4 p, bool &moved) {
    // periodicWrap (GridGPU.cu:138-161), per site
    const float ix = floorf((p.x - box.lo.x) / box.L.x);
    const float iy = floorf((p.y - box.lo.y) / box.L.y);
    const float iz = floorf((p.z - box.lo.z) / box.L.z);
    moved = ix != 0.f || iy != 0.f || iz != 0.f;
    if (moved) {
        p.x = p.x - box.L.x * ix;
        p.y = p.y - box.L.y * iy;
        p.z = p.z - box.L.z * iz;
    }
    return p;
}

// site 0 wrapped into the box (periodicWrap's formula), the other sites put
// at their minimum-image offset from it, so every molecule is stored whole
// (as SETTLE leaves it after every step); the molecule binned by its site 0
__global__ void k_mf_wrap_bin(const MolGridArgs m0, const MolGridArgs *__restrict__ tab) {
    MDX_MG_ARGS;
    if (!M.st->rebuild) return;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M.nmol) return;
    const int4 ix = M.mol_idx[m];
    const int at[4] = {ix.x, ix.y, ix.z, ix.w};
    bool moved;
    const float4 r0 = M.xs[at[0]];
    const float4 p0 = wrap_pos(M.box, r0, moved);
    if (moved) M.xs[at[0]] = p0;
#pragma unroll
    for (int k = 1; k < 4; k++) {
        const float4 r = M.xs[at[k]];
        const float3 d = min_image(M.box, f3(r) - f3(r0));
        const float4 p = make_float4(p0.x + d.x, p0.y + d.y, p0.z + d.z, r.w);
        if (p.x != r.x || p.y != r.y || p.z != r.z) M.xs[at[k]] = p;
    }
    const int c = cell_of_pos(M.g, f3(p0));
    M.cell_of[m] = c;
    atomicAdd(M.cell_count + c, 1u);
}

__global__ void k_mf_scatter(const MolGridArgs m0, const MolGridArgs *__restrict__ tab) {
    MDX_MG_ARGS;
    if (!M.st->rebuild) return;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M.nmol) return;
    const int c = M.cell_of[m];
    const uint32_t slot = atomicAdd(M.cell_fill + c, 1u);
    M.perm_tmp[M.cell_start[c] + slot] = m;
}

// each molecule's slot d, by its rank among the cell's molecule indices
// (deterministic), its four sites into 4d .. 4d+3 of the alternate streams and
// idToIdx rewritten; one thread per site (the four of a molecule each work out
// the rank).  The histogram is cleared for the next build
__global__ void k_mf_gather(const MolGridArgs m0, const MolGridArgs *__restrict__ tab) {
    MDX_MG_ARGS;
    if (!M.st->rebuild) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    for (int c = t; c < M.ncell; c += gridDim.x * blockDim.x) M.cell_count[c] = 0u;
    if (t >= 4 * M.nmol) return;
    const int site = t & 3;
    const int a = M.perm_tmp[t >> 2];
    const int c = M.cell_of[a];
    const uint32_t beg = M.cell_start[c], end = M.cell_start[c + 1];
    const int4 ix = M.mol_idx[a];
    uint32_t d = beg;
    for (uint32_t q = beg; q < end; q++) d += M.perm_tmp[q] < a;
    if (site == 0) M.perm[d] = a;
    const int s = site == 0 ? ix.x : (site == 1 ? ix.y : (site == 2 ? ix.z : ix.w));
    const int o = 4 * (int)d + site;
    M.xs2[o] = M.xs[s];
    M.vs2[o] = M.vs[s];
    M.fs2[o] = M.fs[s];
    M.qs2[o] = M.qs[s];
    const uint32_t id = M.ids[s];
    M.ids2[o] = id;
    M.idToIdx[id] = o;
}

// the sorted streams back into the primary buffers, the positions of this
// build for the skin check, and the molecule maps (molecule perm[d] at slot d)
__global__ void k_mf_copyback(const MolGridArgs m0, const MolGridArgs *__restrict__ tab) {
    MDX_MG_ARGS;
    if (!M.st->rebuild) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 4 * M.nmol) return;
    const float4 p = M.xs2[i];
    M.xs[i] = p;
    M.xs_last[i] = p;
    M.vs[i] = M.vs2[i];
    M.fs[i] = M.fs2[i];
    M.qs[i] = M.qs2[i];
    M.ids[i] = M.ids2[i];
    if ((i & 3) == 0) {
        const int d = i >> 2;
        const int4 nx = make_int4(i, i + 1, i + 2, i + 3);
        M.mol_idx[M.perm[d]] = nx;
        if (M.mol_idx_e3b) M.mol_idx_e3b[M.perm[d]] = nx;
    }
}

CellGrid make_grid(const State &s) {
    CellGrid g;
    g.lo = s.box.lo;
    g.ns = s.grid.ns;
    g.inv_ds = make_float3((float)(s.grid.ns.x / s.box.Ld.x), (float)(s.grid.ns.y / s.box.Ld.y),
                           (float)(s.grid.ns.z / s.box.Ld.z));
    return g;
}

GridArgs grid_args(State &s) {
    GridGPU &gr = s.grid;
    GPUData &d = s.gpd;
    GridArgs A{};
    A.xs = d.xs.p;
    A.vs = d.vs.p;
    A.fs = d.fs.p;
    A.qs = d.qs.p;
    A.ids = d.ids.p;
    A.xs2 = d.xs_alt.p;
    A.vs2 = d.vs_alt.p;
    A.fs2 = d.fs_alt.p;
    A.qs2 = d.qs_alt.p;
    A.ids2 = d.ids_alt.p;
    A.xs_last = d.xs_last_build.p;
    A.idToIdx = d.idToIdx.p;
    A.cell_of = gr.cell_of.p;
    A.cell_count = gr.cell_count.p;
    A.cell_start = gr.cell_start.p;
    A.cell_fill = gr.cell_fill.p;
    A.perm_tmp = gr.perm_tmp.p;
    A.st = s.d_status.p;
    A.box = s.box;
    A.g = make_grid(s);
    A.n = d.n;
    A.ncell = gr.ns.x * gr.ns.y * gr.ns.z;
    A.interval = s.periodicInterval;
    A.skin2q = (float)(s.padding * s.padding) * 0.25f;
    A.view = 0;
    return A;
}

CellGrid mol_grid(const State &s) {
    CellGrid g;
    g.lo = s.box.lo;
    g.ns = s.mf.ns;
    g.inv_ds = make_float3((float)(s.mf.ns.x / s.box.Ld.x), (float)(s.mf.ns.y / s.box.Ld.y),
                           (float)(s.mf.ns.z / s.box.Ld.z));
    return g;
}

MolGridArgs mol_grid_args(State &s) {
    MolForm &mf = s.mf;
    GPUData &d = s.gpd;
    MolGridArgs M{};
    M.xs = d.xs.p;
    M.vs = d.vs.p;
    M.fs = d.fs.p;
    M.qs = d.qs.p;
    M.ids = d.ids.p;
    M.xs2 = d.xs_alt.p;
    M.vs2 = d.vs_alt.p;
    M.fs2 = d.fs_alt.p;
    M.qs2 = d.qs_alt.p;
    M.ids2 = d.ids_alt.p;
    M.xs_last = d.xs_last_build.p;
    M.idToIdx = d.idToIdx.p;
    M.mol_idx = s.rigidFix()->d_mol_idx.p;
    // (FixE3B's map is the identity slot map in this form, never rewritten)
    M.mol_idx_e3b = nullptr;
    M.cell_of = mf.cell_of.p;
    M.cell_count = mf.cell_count.p;
    M.cell_start = mf.cell_start.p;
    M.cell_fill = mf.cell_fill.p;
    M.perm_tmp = mf.perm_tmp.p;
    M.perm = mf.perm.p;
    M.st = s.d_status.p;
    M.box = s.box;
    M.g = mol_grid(s);
    M.nmol = mf.nmol;
    M.ncell = mf.ns.x * mf.ns.y * mf.ns.z;
    return M;
}

// the scan / finish kernels over the molecule grid's cell arrays
GridArgs mol_scan_args(State &s) {
    GridArgs A = grid_args(s);
    A.cell_count = s.mf.cell_count.p;
    A.cell_start = s.mf.cell_start.p;
    A.cell_fill = s.mf.cell_fill.p;
    A.ncell = s.mf.ns.x * s.mf.ns.y * s.mf.ns.z;
    return A;
}

// warps per cell of the list build: as many as the SMs hold at once (28 each),
// to the nearest, four at most.  A small system's build takes as long as its
// fullest cell's warp: 2,048 water sites (729 cells) 74 us with one warp per
// cell, 47 with four; 4,096 molecules (1,728 cells) 46 and, with two, 37;
// 8,000 ions (2,744 cells) 46.5 and 44.3.  Beyond what is resident the cell's
// candidates are only expanded once more: 32,000 particles (13,824 cells) 63
// and 71.
inline int build_parts(int ncell) {
    const int resident = 28 * num_sms();
    return std::min(4, std::max(1, (resident + ncell / 2) / std::max(ncell, 1)));
}

BuildArgs build_args(State &s, const CellGrid &g, float cutsq) {
    GridGPU &gr = s.grid;
    GPUData &d = s.gpd;
    BuildArgs A{};
    A.xs2 = d.xs_alt.p;
    A.vs2 = d.vs_alt.p;
    A.fs2 = d.fs_alt.p;
    A.qs2 = d.qs_alt.p;
    A.ids2 = d.ids_alt.p;
    A.xs = d.xs.p;
    A.vs = d.vs.p;
    A.fs = d.fs.p;
    A.qs = d.qs.p;
    A.ids = d.ids.p;
    A.xs_last = d.xs_last_build.p;
    A.cell_start = gr.cell_start.p;
    A.excl_start = gr.excl_start.p;
    A.excl_ids = gr.excl_ids.p;
    A.excl_win = gr.excl_win.p;
    A.excl_far = gr.excl_far.p;
    A.ljmask = gr.partition ? gr.ljmask.p : nullptr;
    A.counts = gr.counts.p;
    A.counts_int = gr.counts_int.p;
    A.nlist = gr.nlist.p;
    A.st = s.d_status.p;
    A.g = g;
    A.box = s.box;
    A.ncell = g.ns.x * g.ns.y * g.ns.z;
    A.parts = build_parts(A.ncell);
    A.m = gr.m;
    A.use_excl = gr.have_excl ? 1 : 0;
    A.part_q = gr.part_q ? 1 : 0;
    A.cap = gr.cap;
    A.cutsq = cutsq;
    return A;
}

template <int T, int HG, bool COUNT>
auto build_kernel(bool split, bool excl) {
    if constexpr (COUNT) {
        return k_build_cells<T, HG, true, false, false>;
    } else {
        return split ? (excl ? k_build_cells<T, HG, false, true, true> : k_build_cells<T, HG, false, true, false>)
                     : (excl ? k_build_cells<T, HG, false, false, true> : k_build_cells<T, HG, false, false, false>);
    }
}

template <int T, bool COUNT>
void launch_build_hg(int hg, dim3 grid, cudaStream_t st, const BuildArgs &A, const BuildArgs *tab) {
    const bool split = A.ljmask != nullptr, excl = A.use_excl != 0;
    auto k = hg == 4 ? build_kernel<T, 4, COUNT>(split, excl) : build_kernel<T, 2, COUNT>(split, excl);
    if (tab) {
        k<<<grid, kBuildCellsPerBlock * 32, 0, st>>>(A, tab);
        MDX_LAUNCHED();
    } else {
        launch_pdl(k, grid, dim3(kBuildCellsPerBlock * 32), 0, st, A, tab);
    }
}

// grid.x covers ncell (or the largest replica's) cells, one warp each
template <bool COUNT>
void launch_build_any(int team, int hg, dim3 grid, cudaStream_t st, const BuildArgs &A, const BuildArgs *tab) {
    switch (team) {
        case 1: launch_build_hg<1, COUNT>(hg, grid, st, A, tab); break;
        case 2: launch_build_hg<2, COUNT>(hg, grid, st, A, tab); break;
        case 4: launch_build_hg<4, COUNT>(hg, grid, st, A, tab); break;
        case 8: launch_build_hg<8, COUNT>(hg, grid, st, A, tab); break;
        case 16: launch_build_hg<16, COUNT>(hg, grid, st, A, tab); break;
        default: launch_build_hg<32, COUNT>(hg, grid, st, A, tab); break;
    }
}

inline dim3 build_grid(int ncell, int parts, int nrep) {
    return dim3((ncell * parts + kBuildCellsPerBlock - 1) / kBuildCellsPerBlock, nrep);
}

void launch_build(State &s, const CellGrid &g, float cutsq, cudaStream_t st) {
    const BuildArgs A = build_args(s, g, cutsq);
    launch_build_any<false>(s.grid.team, s.grid.home_group, build_grid(A.ncell, A.parts, 1), st, A, nullptr);
}

// the molecule-pair list: rows of 32 lanes, its molecules' site 0 within the
// list radius of site 0.  k_build_cells over the molecule grid: a warp per
// cell expands the cell's candidates once for its two or three molecules.  (A
// block per molecule, a thread per stencil row walking it twice: 60 us at
// 4,096 molecules, 327 us at 32,768.)
constexpr int kMolHomes = 2;  // home molecules tested at once
BuildArgs mol_build_args(State &s) {
    MolForm &mf = s.mf;
    BuildArgs A{};
    A.xs2 = s.gpd.xs_alt.p;
    A.cell_start = mf.cell_start.p;
    A.counts = mf.counts.p;
    A.nlist = mf.list.p;
    A.st = s.d_status.p;
    A.g = mol_grid(s);
    A.box = s.box;
    A.ncell = mf.ns.x * mf.ns.y * mf.ns.z;
    A.parts = build_parts(A.ncell);
    A.m = mf.m;
    A.cap = mf.cap;
    A.cutsq = mf.cut * mf.cut;
    return A;
}

void launch_count(State &s, const CellGrid &g, float cutsq) {
    BuildArgs A = build_args(s, g, cutsq);
    A.use_excl = 0;
    A.ljmask = nullptr;
    A.part_q = 0;
    A.cap = 0;
    launch_build_any<true>(s.grid.team, s.grid.home_group, build_grid(A.ncell, A.parts, 1), s.stream, A, nullptr);
}

}  // namespace

// Exclusion list by bond-graph depth (handleExclusionsDistance /
// generateExclusionList, GridGPU.cu:1377-1518): level d+1 = neighbours of
// level-d atoms that are not closer and not the atom itself; tags 1..3.
int nlist_exclusions(State &s) {
    std::vector<std::pair<int, int>> bonds;
    for (Fix *f : s.fixes) f->getBonds(bonds);
    GridGPU &gr = s.grid;
    gr.have_excl = !bonds.empty();
    gr.h_excl_start.assign(s.atoms.size() + 1, 0);
    gr.h_excl_ids.clear();
    if (!gr.have_excl) return 0;
    const int nid = (int)s.atoms.size();
    std::vector<std::vector<int>> adj(nid);
    for (auto &b : bonds) {
        adj[b.first].push_back(b.second);
        adj[b.second].push_back(b.first);
    }
    std::vector<int> start(nid + 1, 0);
    std::vector<uint32_t> ent;
    std::vector<int> level(nid, -1);  // scratch: depth at which an id was reached
    std::vector<int> touched;
    for (int i = 0; i < nid; i++) {
        touched.clear();
        level[i] = 0;
        touched.push_back(i);
        std::vector<int> frontier{i};
        for (int depth = 1; depth <= 3; depth++) {
            std::vector<int> next;
            for (int a : frontier)
                for (int b : adj[a])
                    if (level[b] < 0) {
                        level[b] = depth;
                        touched.push_back(b);
                        next.push_back(b);
                    }
            std::sort(next.begin(), next.end());
            next.erase(std::unique(next.begin(), next.end()), next.end());
            for (int b : next) ent.push_back((uint32_t)b | ((uint32_t)depth << 30));
            frontier.swap(next);
        }
        for (int t : touched) level[t] = -1;
        start[i + 1] = (int)ent.size();
        gr.max_excl = std::max(gr.max_excl, start[i + 1] - start[i]);
    }
    std::vector<ulonglong2> win(nid, make_ulonglong2(0ull, 0ull));
    std::vector<uint8_t> far(nid, 0);
    for (int i = 0; i < nid; i++)
        for (int e = start[i]; e < start[i + 1]; e++) {
            const long long d = (long long)(ent[e] & kExclMask) - i + 32;
            const uint32_t depth = ent[e] >> 30;
            if (d < 0 || d >= 64) {
                far[i] = 1;
                continue;
            }
            if (depth & 1u) win[i].x |= 1ull << d;
            if (depth & 2u) win[i].y |= 1ull << d;
        }
    if (int e = gr.excl_win.alloc(nid)) return e;
    if (int e = gr.excl_far.alloc(nid)) return e;
    MDX_CUDA_TRY(cudaMemcpy(gr.excl_win.p, win.data(), nid * sizeof(ulonglong2), cudaMemcpyHostToDevice));
    MDX_CUDA_TRY(cudaMemcpy(gr.excl_far.p, far.data(), nid * sizeof(uint8_t), cudaMemcpyHostToDevice));
    gr.h_excl_start = start;
    gr.h_excl_ids = ent;
    if (int e = gr.excl_start.alloc(start.size())) return e;
    if (int e = gr.excl_ids.alloc(ent.size())) return e;
    MDX_CUDA_TRY(cudaMemcpy(gr.excl_start.p, start.data(), start.size() * sizeof(int), cudaMemcpyHostToDevice));
    MDX_CUDA_TRY(cudaMemcpy(gr.excl_ids.p, ent.data(), ent.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    return 0;
}

// Which listed pairs can interact: bit tj of ljmask[ti] is set when the pair
// fix's evaluator can give (ti, tj) a force (eps != 0; eps14 != 0 for
// LJCHARMM; C != 0 for TICG); with a charge fix (Ewald or DSF), pairs with
// q_i q_j != 0 also interact.  Everything else contributes exactly zero
// force, energy and virial in compute_force_iso (the pair evaluators scale by
// eps or C, the charge evaluators by q_i q_j) and is kept at the back of the
// row.
int nlist_set_interactions(State &s) {
    GridGPU &gr = s.grid;
    FixPair *pf = s.pairFix();
    const int nt = (int)s.species.size();
    gr.partition = false;
    gr.part_q = false;
    if (!pf || nt > 32 || pf->h_params.size() != (size_t)pf->nparam() * nt * nt) return 0;
    std::vector<uint32_t> mask(nt, 0u);
    for (int a = 0; a < nt; a++)
        for (int b = 0; b < nt; b++)
            if (pf->pairActive(a, b)) mask[a] |= 1u << b;
    if (int e = gr.ljmask.alloc(nt)) return e;
    MDX_CUDA_TRY(cudaMemcpy(gr.ljmask.p, mask.data(), nt * sizeof(uint32_t), cudaMemcpyHostToDevice));
    gr.part_q = pf->chargeFix != nullptr || pf->dsfFix != nullptr;
    // without charges and with no zero pair there is nothing to split off
    bool all = true;
    for (int a = 0; a < nt; a++) all = all && mask[a] == (nt == 32 ? 0xffffffffu : (1u << nt) - 1u);
    gr.partition = gr.part_q || !all;
    return 0;
}

// Grid set-up (GridGPU::setBounds, GridGPU.cu:46-66): cells of width
// >= cut/m instead of >= cut, m chosen below.
int nlist_init(State &s) {
    GridGPU &gr = s.grid;
    gr.cut = (float)((double)(float)s.maxRCut() + s.padding);
    gr.skin = (float)s.padding;
    // minimum image: one periodic image of a pair at most can lie within cut
    if (2.0 * (double)gr.cut >= std::min(s.box.Ld.x, std::min(s.box.Ld.y, s.box.Ld.z))) {
        set_error(MDX_ERR_UNSUPPORTED, "neighbour cutoff %g (rCut + padding) must be below half the box (%g %g %g)",
                  (double)gr.cut, s.box.Ld.x, s.box.Ld.y, s.box.Ld.z);
        return MDX_ERR_UNSUPPORTED;
    }
    // cells of at least cut/m, m as large as keeps a mean of 2 atoms per
    // cell (finer cells trim the candidate volume toward the cutoff sphere).
    // A (2m+1)-cell stencil row wraps the box at most once when there are
    // >= 2m cells per side; a cell it visits under two images holds at most
    // one image within cut < L/2.  m = 1 needs 3 cells per side.
    if (s.gridStencil < 0 || s.gridStencil > kStencilMax) {
        set_error(MDX_ERR_ARG, "gridStencil must be 0 (automatic) or 1..%d (got %d)", kStencilMax, s.gridStencil);
        return MDX_ERR_ARG;
    }
    int m = s.gridStencil > 0 ? s.gridStencil : kStencilMax;
    int3 ns;
    for (;; m--) {
        if (m == 0) {
            set_error(MDX_ERR_UNSUPPORTED, "box (%g %g %g) too small for neighbour cutoff %g: need >= 3 cells per side",
                      s.box.Ld.x, s.box.Ld.y, s.box.Ld.z, (double)gr.cut);
            return MDX_ERR_UNSUPPORTED;
        }
        double w = (double)gr.cut / m * (1.0 + 1e-5);
        ns = make_int3((int)(s.box.Ld.x / w), (int)(s.box.Ld.y / w), (int)(s.box.Ld.z / w));
        const int need = std::max(3, 2 * m);
        if (ns.x < need || ns.y < need || ns.z < need) continue;
        if (m == 1 || s.gridStencil > 0 || (double)s.gpd.n >= 2.0 * ns.x * ns.y * ns.z) break;
    }
    if (s.gpd.n >= (1 << kCandIdxBits)) {
        set_error(MDX_ERR_UNSUPPORTED, "neighbour list build limited to %d atoms (got %d)", 1 << kCandIdxBits, s.gpd.n);
        return MDX_ERR_UNSUPPORTED;
    }
    gr.m = m;
    gr.ns = ns;
    int ncell = ns.x * ns.y * ns.z;
    // list build: home atoms tested two at a time, also where cells hold more.
    // Water (split rows, exclusions) is slower four at a time: 160 us a build
    // against 117 at six atoms in a cell, 184 against 162 at 32.  Where the
    // grid chosen above puts four to sixteen LJ atoms in a cell it makes
    // little difference, two against four at density 0.2: 28.1, 28.1 us (4,000
    // atoms), 54.7, 54.7 (32,000), 242, 248 (256,000); at 0.4: 36.3, 36.2;
    // 64.9, 69.0; 267, 261
    if (s.gridHomeGroup != 0 && s.gridHomeGroup != 2 && s.gridHomeGroup != 4) {
        set_error(MDX_ERR_ARG, "gridHomeGroup must be 0 (automatic), 2 or 4 (got %d)", s.gridHomeGroup);
        return MDX_ERR_ARG;
    }
    gr.home_group = s.gridHomeGroup ? s.gridHomeGroup : 2;
    if (int e = gr.cell_start.alloc(ncell + 1)) return e;
    if (int e = gr.cell_count.alloc(ncell)) return e;
    if (int e = gr.cell_fill.alloc(ncell)) return e;
    MDX_CUDA_TRY(cudaMemsetAsync(gr.cell_count.p, 0, ncell * sizeof(uint32_t), s.stream));
    const int n = s.gpd.n;
    if (int e = gr.cell_of.alloc(n)) return e;
    if (int e = gr.perm_tmp.alloc(n)) return e;
    if (int e = gr.counts.alloc(n)) return e;
    if (int e = gr.counts_int.alloc(n)) return e;
    if (s.nThreadPerAtom > 0) {
        gr.team = s.nThreadPerAtom;
    } else {
        // density * list volume -> mean neighbours; a wide team for long rows
        // (water, 558 entries: 32 lanes measured 11 % faster than 16 in the
        // pair kernel, which reads only the interacting front of each row)
        double vol = s.box.Ld.x * s.box.Ld.y * s.box.Ld.z;
        double nbar = n / vol * 4.18879 * (double)gr.cut * gr.cut * gr.cut;
        gr.team = nbar > 400 ? 32 : (nbar > 256 ? 16 : (nbar > 128 ? 8 : (nbar > 48 ? 4 : 2)));
        // a small system leaves lanes idle and waits for each row's chain of
        // gathers: wider teams while they fit the SMs, fewer beside a P3M
        // chain.  Measured on B200, us per step at team 4, 8, 16, 32 -- LJ
        // fluid (NVE) 1,500: 9.4 7.0 5.9 5.3; 4,000: 9.8 7.4 6.6 6.8; 6,000:
        // 10.2 7.8 7.2 8.2; 8,000: 10.3 8.0 8.0 9.2; 16,000: 13.2 11.7 12.9
        // 15.8; 32,000: 15.6 16.2 18.0 24.1; salt with P3M, before the steps
        // were joined, 2,000: 28.8 26.6 26.6 26.5; 8,000: 38.7 35.2 38.0 40.6;
        // 24,000: 65.6 69.4 70.7.  The rule takes the best of these but at
        // 4,000 (32 lanes, 3 % over 16)
        const double lanes = (s.ewaldFix() ? 640.0 : 880.0) * num_sms();
        while (gr.team < 32 && gr.team < nbar && 2.0 * gr.team * n <= lanes) gr.team *= 2;
    }
    if (gr.team != 1 && gr.team != 2 && gr.team != 4 && gr.team != 8 && gr.team != 16 && gr.team != 32) {
        set_error(MDX_ERR_ARG, "nThreadPerAtom must be 1,2,4,8,16 or 32 (got %d)", gr.team);
        return MDX_ERR_ARG;
    }
    // a state prepared again keeps its list buffer, unless the rows it was
    // sized for changed: with another team a capacity that is no multiple of
    // it makes neighbouring rows overlap and the last one pass the buffer's
    // end, and more atoms or a longer cutoff need more room
    if (gr.cap_team != gr.team || gr.cap_n != n || gr.cap_cut != gr.cut) {
        gr.cap = 0;
        gr.cap_team = gr.team;
        gr.cap_n = n;
        gr.cap_cut = gr.cut;
    }
    return nlist_exclusions(s);
}

// GridGPU::periodicBoundaryConditions (GridGPU.cu:824-1103).  conditional:
// run the check kernel that decides on the device (graph mode); otherwise
// the rebuild is forced (force=true) or decided by the same check.
// bstream (optional): the list build, the E3B molecule list and k_finish go
// to that stream after the sort, so the caller can run the step's first half
// and the P3M chain beside them; it waits on s.ev_join[2] (recorded at the
// end of bstream) before anything that reads the lists.
static int nlist_rebuild_mf(State &s, bool force, cudaStream_t bstream);

int nlist_rebuild(State &s, bool force, bool conditional, cudaStream_t bstream) {
    if (s.mf.on) return nlist_rebuild_mf(s, force, bstream);
    GridGPU &gr = s.grid;
    GPUData &d = s.gpd;
    const int n = d.n;
    const int ncell = gr.ns.x * gr.ns.y * gr.ns.z;
    const CellGrid g = make_grid(s);
    const float cutsq = gr.cut * gr.cut;
    (void)conditional;
    const GridArgs A = grid_args(s);
    const int nb = (n + 255) / 256;
    const GridArgs *nt = nullptr;
    MDX_CUDA_TRY(launch_pdl(k_check, dim3(nb), dim3(256), 0, s.stream, A, nt, force ? 1 : 0));
    MDX_CUDA_TRY(launch_pdl(k_wrap_bin, dim3(nb), dim3(256), 0, s.stream, A, nt));
    MDX_CUDA_TRY(launch_pdl(k_scan_cells, dim3(scan_blocks(A.ncell)), dim3(kScanThreads), 0, s.stream, A, nt));
    MDX_CUDA_TRY(launch_pdl(k_scatter, dim3(nb), dim3(256), 0, s.stream, A, nt));
    MDX_CUDA_TRY(launch_pdl(k_gather, dim3(nb), dim3(256), 0, s.stream, A, nt));
    MDX_CUDA_TRY(launch_pdl(k_copyback, dim3(nb), dim3(256), 0, s.stream, A, nt));
    // molecule maps of the fixes that keep atom indices
    if (FixRigid *r = s.rigidFix()) {
        if (int e = rigid_update_maps(s, *r, true)) return e;
    }
    if (gr.cap == 0) {
        // first build: size the per-atom capacity from a counting sweep
        MDX_CUDA_TRY(cudaMemsetAsync(&s.d_status.p->max_neighbors, 0, sizeof(uint32_t), s.stream));
        launch_count(s, g, cutsq);
        uint32_t mx = 0;
        MDX_CUDA_TRY(cudaMemcpyAsync(&mx, &s.d_status.p->max_neighbors, sizeof(uint32_t), cudaMemcpyDeviceToHost,
                                     s.stream));
        MDX_CUDA_TRY(cudaStreamSynchronize(s.stream));
        int c = (int)(mx * 1.35 + 32);
        c = (c + gr.team - 1) / gr.team * gr.team;
        gr.cap = c;
        size_t groups = (size_t)(n + (32 / gr.team) - 1) / (32 / gr.team);
        if (int e = gr.nlist.alloc(groups * (size_t)c * (32 / gr.team))) return e;
    }
    cudaStream_t bs = s.stream;
    if (bstream) {
        MDX_CUDA_TRY(cudaEventRecord(s.ev_sorted, s.stream));
        MDX_CUDA_TRY(cudaStreamWaitEvent(bstream, s.ev_sorted, 0));
        bs = bstream;
    }
    launch_build(s, g, cutsq, bs);
    if (FixE3B *e3 = s.e3bFix()) {
        if (int e = e3b_build_list(s, *e3, true, bs)) return e;
    }
    MDX_CUDA_TRY(launch_pdl(k_finish, dim3(1), dim3(1), 0, bs, A, (const GridArgs *)nullptr));
    if (bs != s.stream) MDX_CUDA_TRY(cudaEventRecord(s.ev_join[2], bs));
    gr.built = true;
    return 0;
}

// a prepared state's list in rows for another number of lanes per atom
int nlist_set_team(State &s, int team) {
    s.grid.team = s.grid.cap_team = team;
    s.grid.cap = 0;
    s.box_gen++;
    return nlist_rebuild(s, true, false);
}

// The molecule form's rebuild group: the same skin check, then the sort by
// molecule, then (on bstream when given, beside the step's first half) the
// molecule-pair list and the E3B molecule list cut from it.
static int nlist_rebuild_mf(State &s, bool force, cudaStream_t bstream) {
    const GridArgs A = grid_args(s);
    const GridArgs Am = mol_scan_args(s);
    const MolGridArgs M = mol_grid_args(s);
    const GridArgs *nt = nullptr;
    const MolGridArgs *mnt = nullptr;
    const int nb_atoms = (s.gpd.n + 255) / 256;
    const int nb_mol = (M.nmol + 255) / 256;
    MDX_CUDA_TRY(launch_pdl(k_check, dim3(nb_atoms), dim3(256), 0, s.stream, A, nt, force ? 1 : 0));
    MDX_CUDA_TRY(launch_pdl(k_mf_wrap_bin, dim3(nb_mol), dim3(256), 0, s.stream, M, mnt));
    MDX_CUDA_TRY(launch_pdl(k_scan_cells, dim3(scan_blocks(Am.ncell)), dim3(kScanThreads), 0, s.stream, Am, nt));
    MDX_CUDA_TRY(launch_pdl(k_mf_scatter, dim3(nb_mol), dim3(256), 0, s.stream, M, mnt));
    MDX_CUDA_TRY(launch_pdl(k_mf_gather, dim3((4 * M.nmol + 255) / 256), dim3(256), 0, s.stream, M, mnt));
    MDX_CUDA_TRY(launch_pdl(k_mf_copyback, dim3((4 * M.nmol + 255) / 256), dim3(256), 0, s.stream, M, mnt));
    cudaStream_t bs = s.stream;
    if (bstream) {
        MDX_CUDA_TRY(cudaEventRecord(s.ev_sorted, s.stream));
        MDX_CUDA_TRY(cudaStreamWaitEvent(bstream, s.ev_sorted, 0));
        bs = bstream;
    }
    MDX_CUDA_TRY(launch_pdl(k_build_cells<32, kMolHomes, false, false, false, 4>, build_grid(M.ncell, mol_build_args(s).parts, 1),
                            dim3(kBuildCellsPerBlock * 32), 0, bs, mol_build_args(s), (const BuildArgs *)nullptr));
    if (FixE3B *e3 = s.e3bFix()) {
        if (int e = e3b_build_list_mf(s, *e3, bs)) return e;
    }
    MDX_CUDA_TRY(launch_pdl(k_finish, dim3(1), dim3(1), 0, bs, Am, nt));
    if (bs != s.stream) MDX_CUDA_TRY(cudaEventRecord(s.ev_join[2], bs));
    s.grid.built = true;
    return 0;
}

// The per-site list (the reference's GridGPU list) of the current positions
// built into the sort's alternate buffers only: the molecule form's primary
// streams, idToIdx, molecule maps and skin-check positions are untouched.
// The list's atom indices refer to that sorted copy (ids_alt holds its ids).
int nlist_build_atoms_view(State &s) {
    GridGPU &gr = s.grid;
    const int n = s.gpd.n;
    const CellGrid g = make_grid(s);
    const float cutsq = gr.cut * gr.cut;
    GridArgs A = grid_args(s);
    A.view = 1;
    const int nb = (n + 255) / 256;
    const int ncell = gr.ns.x * gr.ns.y * gr.ns.z;
    const GridArgs *nt = nullptr;
    MDX_CUDA_TRY(launch_pdl(k_check, dim3(nb), dim3(256), 0, s.stream, A, nt, 1));
    MDX_CUDA_TRY(launch_pdl(k_wrap_bin, dim3(nb), dim3(256), 0, s.stream, A, nt));
    MDX_CUDA_TRY(launch_pdl(k_scan_cells, dim3(scan_blocks(A.ncell)), dim3(kScanThreads), 0, s.stream, A, nt));
    MDX_CUDA_TRY(launch_pdl(k_scatter, dim3(nb), dim3(256), 0, s.stream, A, nt));
    MDX_CUDA_TRY(launch_pdl(k_gather, dim3(nb), dim3(256), 0, s.stream, A, nt));
    if (gr.cap == 0) {
        MDX_CUDA_TRY(cudaMemsetAsync(&s.d_status.p->max_neighbors, 0, sizeof(uint32_t), s.stream));
        launch_count(s, g, cutsq);
        uint32_t mx = 0;
        MDX_CUDA_TRY(cudaMemcpyAsync(&mx, &s.d_status.p->max_neighbors, sizeof(uint32_t), cudaMemcpyDeviceToHost,
                                     s.stream));
        MDX_CUDA_TRY(cudaStreamSynchronize(s.stream));
        int c = (int)(mx * 1.35 + 32);
        c = (c + gr.team - 1) / gr.team * gr.team;
        gr.cap = c;
        size_t groups = (size_t)(n + (32 / gr.team) - 1) / (32 / gr.team);
        if (int e = gr.nlist.alloc(groups * (size_t)c * (32 / gr.team))) return e;
    }
    launch_build(s, g, cutsq, s.stream);
    MDX_CUDA_TRY(launch_pdl(k_finish, dim3(1), dim3(1), 0, s.stream, A, nt));
    return 0;
}

// Molecule form set-up (see MolForm): decides whether the system allows it
// and sizes its grid and list.  pairForm 1 keeps the per-site form; 2 makes
// an unsuitable system an error; 0 takes the molecule form when it can.
int molform_init(State &s) {
    MolForm &mf = s.mf;
    mf.on = false;
    if (s.pairForm == 1) return 0;
    auto refuse = [&](const char *why) -> int {
        if (s.pairForm != 2) return 0;
        set_error(MDX_ERR_UNSUPPORTED, "pairForm 2 (molecule form) not possible: %s", why);
        return MDX_ERR_UNSUPPORTED;
    };
    FixRigid *r = s.rigidFix();
    FixPair *pf = s.pairFix();
    if (!r || !r->foursite) return refuse("needs FixRigid with four-site molecules");
    if (!pf) return refuse("needs a pair fix");
    if (pf->lj_kind != 1 && pf->lj_kind != 2) return refuse("the molecule form evaluates LJ/cut or WCA");
    if (s.dsfFix()) return refuse("the molecule form evaluates Ewald real-space charges");
    if (has_free_atoms(s)) return refuse("every atom must belong to a rigid molecule");
    if (FixE3B *e3 = s.e3bFix())
        if (!e3->side_ok) return refuse("FixE3B's molecules must be FixRigid's, in the same order");
    const int nmol = (int)r->mol_ids.size();
    if (nmol == 0) return refuse("no molecules");
    auto site = [&](const int4 &m, int k) { return k == 0 ? m.x : (k == 1 ? m.y : (k == 2 ? m.z : m.w)); };
    // every molecule alike: site types and charges (as stored, FP32)
    const int4 m0 = r->mol_ids[0];
    for (int k = 0; k < 4; k++) {
        mf.type[k] = s.atoms[site(m0, k)].type;
        mf.q[k] = (float)s.atoms[site(m0, k)].q;
    }
    for (const int4 &m : r->mol_ids)
        for (int k = 0; k < 4; k++) {
            const HostAtom &a = s.atoms[site(m, k)];
            if (a.type != mf.type[k] || (float)a.q != mf.q[k]) return refuse("molecules differ in site types or charges");
        }
    // exclusions only inside a molecule, by the same depth in every molecule
    const GridGPU &gr = s.grid;
    std::vector<int> site_of(s.atoms.size(), -1), mol_of(s.atoms.size(), -1);
    for (int mi = 0; mi < nmol; mi++)
        for (int k = 0; k < 4; k++) {
            site_of[site(r->mol_ids[mi], k)] = k;
            mol_of[site(r->mol_ids[mi], k)] = mi;
        }
    for (int k = 0; k < 16; k++) mf.depth[k] = 0;
    bool first = true;
    for (int mi = 0; mi < nmol; mi++) {
        int dep[16] = {0};
        for (int k = 0; k < 4; k++) {
            const int id = site(r->mol_ids[mi], k);
            if (!gr.have_excl) break;
            for (int e = gr.h_excl_start[id]; e < gr.h_excl_start[id + 1]; e++) {
                const int o = (int)(gr.h_excl_ids[e] & kExclMask);
                if (mol_of[o] != mi) return refuse("an exclusion joins two molecules");
                dep[4 * k + site_of[o]] = (int)(gr.h_excl_ids[e] >> 30);
            }
        }
        if (first) {
            for (int k = 0; k < 16; k++) mf.depth[k] = dep[k];
            first = false;
        } else {
            for (int k = 0; k < 16; k++)
                if (dep[k] != mf.depth[k]) return refuse("molecules differ in their exclusions");
        }
    }
    // site 0 to any other site: the rigid geometry (+ a margin for the
    // FP32 positions SETTLE leaves)
    const double dmax = std::max(r->rc.r_OH, r->rc.r_OM) + 1e-3;
    const double pair_cut = (double)s.maxRCut();
    const double cut = pair_cut + s.padding + 2.0 * dmax;
    const double Lmin = std::min(s.box.Ld.x, std::min(s.box.Ld.y, s.box.Ld.z));
    if (2.0 * cut >= Lmin) return refuse("the molecule list radius must stay below half the box");
    // a site pair within the pair cutoff lies within pair_cut + 4 dmax under
    // the site-0 image shift, which must be the unique image within L/2
    if (2.0 * (pair_cut + 4.0 * dmax) >= Lmin) return refuse("box too small for one image shift per molecule pair");
    if (2.0 * dmax >= (double)gr.cut) return refuse("a molecule must lie within the neighbour cutoff");
    // cells >= cut / m with at least 2m + 1 per side; the finest such grid
    // that keeps a mean of two molecules per cell
    int m = 3;
    int3 ns{0, 0, 0};
    for (;; m--) {
        if (m == 0) return refuse("box too small for the molecule grid");
        const double w = cut / m * (1.0 + 1e-5);
        ns = make_int3((int)(s.box.Ld.x / w), (int)(s.box.Ld.y / w), (int)(s.box.Ld.z / w));
        if (ns.x < 2 * m + 1 || ns.y < 2 * m + 1 || ns.z < 2 * m + 1) continue;
        if (m == 1 || (double)nmol >= 2.0 * ns.x * ns.y * ns.z) break;
    }
    mf.m = m;
    mf.ns = ns;
    mf.nmol = nmol;
    mf.dmax = (float)dmax;
    mf.cut = (float)cut;
    mf.far = (float)(pair_cut + 2.0 * dmax);
    mf.team = 32;  // one warp per molecule in the pair kernel: each row is contiguous
    const double vol = s.box.Ld.x * s.box.Ld.y * s.box.Ld.z;
    const double nbar = nmol / vol * 4.18879 * cut * cut * cut;
    mf.cap = ((int)(1.5 * nbar + 64) + mf.team - 1) / mf.team * mf.team;
    const int ncell = ns.x * ns.y * ns.z;
    if (int e = mf.cell_start.alloc(ncell + 1)) return e;
    if (int e = mf.cell_count.alloc(ncell)) return e;
    if (int e = mf.cell_fill.alloc(ncell)) return e;
    MDX_CUDA_TRY(cudaMemsetAsync(mf.cell_count.p, 0, ncell * sizeof(uint32_t), s.stream));
    if (int e = mf.cell_of.alloc(nmol)) return e;
    if (int e = mf.perm_tmp.alloc(nmol)) return e;
    if (int e = mf.perm.alloc(nmol)) return e;
    if (int e = mf.counts.alloc(nmol)) return e;
    const int G = 32 / mf.team;
    const size_t groups = (size_t)(nmol + G - 1) / G;
    if (int e = mf.list.alloc(groups * (size_t)mf.cap * G)) return e;
    // the sort reads the molecule maps first: after an upload every atom sits
    // at index == id, so the maps are the molecules' ids
    MDX_CUDA_TRY(cudaMemcpy(r->d_mol_idx.p, r->mol_ids.data(), nmol * sizeof(int4), cudaMemcpyHostToDevice));
    // E3B works by slot in this form (its molecules are FixRigid's): its map
    // is the identity slot map, slot k at sites 4k .. 4k+3
    if (FixE3B *e3 = s.e3bFix()) {
        std::vector<int4> ident(nmol);
        for (int k = 0; k < nmol; k++) ident[k] = make_int4(4 * k, 4 * k + 1, 4 * k + 2, 4 * k + 3);
        MDX_CUDA_TRY(cudaMemcpy(e3->d_mol_idx.p, ident.data(), nmol * sizeof(int4), cudaMemcpyHostToDevice));
    }
    mf.on = true;
    return 0;
}

// the box changed size (a barostat): the cell grids keep their stencil
// widths m and take as many cells per side as the new box holds at that
// width (cells never narrower than the list radius / m); the caller forces a
// rebuild.  The minimum-image and stencil conditions of nlist_init and
// molform_init are checked again.
// a box that grew without bound (a barostat run away) ends the run with an
// error instead of an overflowing grid
static int grid_cells_fit(int3 ns) {
    const long long n = (long long)ns.x * ns.y * ns.z;
    if (n > (1LL << 27)) {
        set_error(MDX_ERR_UNSUPPORTED, "the box grew to %d x %d x %d neighbour cells (more than 2^27)", ns.x, ns.y,
                  ns.z);
        return MDX_ERR_UNSUPPORTED;
    }
    return 0;
}

int nlist_box_changed(State &s) {
    GridGPU &gr = s.grid;
    const double Lmin = std::min(s.box.Ld.x, std::min(s.box.Ld.y, s.box.Ld.z));
    if (2.0 * (double)gr.cut >= Lmin) {
        set_error(MDX_ERR_UNSUPPORTED, "the box shrank below twice the neighbour cutoff %g", (double)gr.cut);
        return MDX_ERR_UNSUPPORTED;
    }
    {
        const double w = (double)gr.cut / gr.m * (1.0 + 1e-5);
        const int3 ns = make_int3((int)(s.box.Ld.x / w), (int)(s.box.Ld.y / w), (int)(s.box.Ld.z / w));
        const int need = std::max(3, 2 * gr.m);
        if (ns.x < need || ns.y < need || ns.z < need) {
            set_error(MDX_ERR_UNSUPPORTED, "the box shrank below the neighbour grid's %d cells per side", need);
            return MDX_ERR_UNSUPPORTED;
        }
        if (int e = grid_cells_fit(ns)) return e;
        const int ncell = ns.x * ns.y * ns.z;
        if (int e = gr.cell_start.alloc(ncell + 1)) return e;
        if (int e = gr.cell_count.alloc(ncell)) return e;
        if (int e = gr.cell_fill.alloc(ncell)) return e;
        MDX_CUDA_TRY(cudaMemsetAsync(gr.cell_count.p, 0, ncell * sizeof(uint32_t), s.stream));
        gr.ns = ns;
    }
    if (s.mf.on) {
        MolForm &mf = s.mf;
        if (2.0 * (double)mf.cut >= Lmin) {
            set_error(MDX_ERR_UNSUPPORTED, "the box shrank below twice the molecule list radius %g", (double)mf.cut);
            return MDX_ERR_UNSUPPORTED;
        }
        const double w = (double)mf.cut / mf.m * (1.0 + 1e-5);
        const int3 ns = make_int3((int)(s.box.Ld.x / w), (int)(s.box.Ld.y / w), (int)(s.box.Ld.z / w));
        if (ns.x < 2 * mf.m + 1 || ns.y < 2 * mf.m + 1 || ns.z < 2 * mf.m + 1) {
            set_error(MDX_ERR_UNSUPPORTED, "the box shrank below the molecule grid's %d cells per side", 2 * mf.m + 1);
            return MDX_ERR_UNSUPPORTED;
        }
        if (int e = grid_cells_fit(ns)) return e;
        const int ncell = ns.x * ns.y * ns.z;
        if (int e = mf.cell_start.alloc(ncell + 1)) return e;
        if (int e = mf.cell_count.alloc(ncell)) return e;
        if (int e = mf.cell_fill.alloc(ncell)) return e;
        MDX_CUDA_TRY(cudaMemsetAsync(mf.cell_count.p, 0, ncell * sizeof(uint32_t), s.stream));
        mf.ns = ns;
    }
    return 0;
}

// batched replicas: the same group, one launch per kernel for all replicas
// of a form (blockIdx.y = replica of that form); every kernel returns at once
// for a replica whose skin check did not fire.  Tables are built at prepare,
// before any capture.
int batch_nlist_tables(Batch &b) {
    const int R = (int)b.reps.size();
    std::vector<GridArgs> hg(R);
    for (int r = 0; r < R; r++) hg[r] = grid_args(*b.reps[r]);
    if (int e = b.tab_grid.alloc(R * sizeof(GridArgs))) return e;
    MDX_CUDA_TRY(cudaMemcpy(b.tab_grid.p, hg.data(), R * sizeof(GridArgs), cudaMemcpyHostToDevice));
    const int P = (int)b.ps.size();
    if (P) {
        std::vector<GridArgs> hp(P);
        std::vector<BuildArgs> hb(P);
        for (int q = 0; q < P; q++) {
            State &s = *b.reps[b.ps[q]];
            hp[q] = hg[b.ps[q]];
            hb[q] = build_args(s, make_grid(s), s.grid.cut * s.grid.cut);
            hb[q].parts = build_parts(b.max_cell_ps * P);
            // one list-build kernel serves the batch: its exclusion and
            // front/back split forms are compile-time, so they must agree
            if ((hb[q].use_excl != 0) != (hb[0].use_excl != 0) ||
                (hb[q].ljmask != nullptr) != (hb[0].ljmask != nullptr)) {
                set_error(MDX_ERR_UNSUPPORTED,
                          "batched replicas must agree on exclusions and on the interacting-pair split (replica %d)",
                          b.ps[q]);
                return MDX_ERR_UNSUPPORTED;
            }
        }
        if (int e = b.tab_grid_ps.alloc(P * sizeof(GridArgs))) return e;
        if (int e = b.tab_build.alloc(P * sizeof(BuildArgs))) return e;
        MDX_CUDA_TRY(cudaMemcpy(b.tab_grid_ps.p, hp.data(), P * sizeof(GridArgs), cudaMemcpyHostToDevice));
        MDX_CUDA_TRY(cudaMemcpy(b.tab_build.p, hb.data(), P * sizeof(BuildArgs), cudaMemcpyHostToDevice));
    }
    const int Q = (int)b.mfi.size();
    if (Q) {
        std::vector<MolGridArgs> hm(Q);
        std::vector<GridArgs> hs(Q);
        std::vector<BuildArgs> hb(Q);
        b.max_mcell = 0;
        for (int q = 0; q < Q; q++) {
            State &s = *b.reps[b.mfi[q]];
            hm[q] = mol_grid_args(s);
            hs[q] = mol_scan_args(s);
            hb[q] = mol_build_args(s);
            b.max_mcell = std::max(b.max_mcell, hs[q].ncell);
        }
        for (BuildArgs &a : hb) a.parts = build_parts(b.max_mcell * Q);
        if (int e = b.tab_molgrid.alloc(Q * sizeof(MolGridArgs))) return e;
        if (int e = b.tab_molscan.alloc(Q * sizeof(GridArgs))) return e;
        if (int e = b.tab_molbuild.alloc(Q * sizeof(BuildArgs))) return e;
        MDX_CUDA_TRY(cudaMemcpy(b.tab_molbuild.p, hb.data(), Q * sizeof(BuildArgs), cudaMemcpyHostToDevice));
        MDX_CUDA_TRY(cudaMemcpy(b.tab_molgrid.p, hm.data(), Q * sizeof(MolGridArgs), cudaMemcpyHostToDevice));
        MDX_CUDA_TRY(cudaMemcpy(b.tab_molscan.p, hs.data(), Q * sizeof(GridArgs), cudaMemcpyHostToDevice));
    }
    return 0;
}

// the per-site replicas' sort and list build (nlist_rebuild's kernels)
static void batch_rebuild_sites(Batch &b, cudaStream_t st) {
    const int P = (int)b.ps.size();
    const GridArgs *tg = reinterpret_cast<const GridArgs *>(b.tab_grid_ps.p);
    const BuildArgs *tb = reinterpret_cast<const BuildArgs *>(b.tab_build.p);
    State &s0 = *b.reps[b.ps[0]];
    GridArgs A = grid_args(s0);  // sizing only: the kernels read tab
    A.n = b.max_n_ps;
    A.ncell = b.max_cell_ps;
    BuildArgs B = build_args(s0, make_grid(s0), s0.grid.cut * s0.grid.cut);
    B.ncell = b.max_cell_ps;
    const dim3 nb((b.max_n_ps + 255) / 256, P);
    k_wrap_bin<<<nb, 256, 0, st>>>(A, tg);
    k_scan_cells<<<dim3(scan_blocks(A.ncell), P), kScanThreads, 0, st>>>(A, tg);
    k_scatter<<<nb, 256, 0, st>>>(A, tg);
    k_gather<<<nb, 256, 0, st>>>(A, tg);
    k_copyback<<<nb, 256, 0, st>>>(A, tg);
    int hg = 2;
    for (int r : b.ps) hg = std::max(hg, b.reps[r]->grid.home_group);
    launch_build_any<false>(s0.grid.team, hg, build_grid(b.max_cell_ps, build_parts(b.max_cell_ps * P), P), st, B, tb);
    g_launches += 5;
}

// the molecule-form replicas' sort by molecule and molecule-pair list
// (nlist_rebuild_mf's kernels)
static void batch_rebuild_mols(Batch &b, cudaStream_t st) {
    const int Q = (int)b.mfi.size();
    const GridArgs *ts = reinterpret_cast<const GridArgs *>(b.tab_molscan.p);
    const MolGridArgs *tm = reinterpret_cast<const MolGridArgs *>(b.tab_molgrid.p);
    State &s0 = *b.reps[b.mfi[0]];
    GridArgs Am = mol_scan_args(s0);  // sizing only: the kernels read the tables
    Am.ncell = b.max_mcell;
    MolGridArgs M = mol_grid_args(s0);
    M.nmol = b.max_mol_mf;
    M.ncell = b.max_mcell;
    const int nb_mol = (b.max_mol_mf + 255) / 256, nb_site = (4 * b.max_mol_mf + 255) / 256;
    k_mf_wrap_bin<<<dim3(nb_mol, Q), 256, 0, st>>>(M, tm);
    k_scan_cells<<<dim3(scan_blocks(Am.ncell), Q), kScanThreads, 0, st>>>(Am, ts);
    k_mf_scatter<<<dim3(nb_mol, Q), 256, 0, st>>>(M, tm);
    k_mf_gather<<<dim3(nb_site, Q), 256, 0, st>>>(M, tm);
    k_mf_copyback<<<dim3(nb_site, Q), 256, 0, st>>>(M, tm);
    k_build_cells<32, kMolHomes, false, false, false, 4><<<build_grid(b.max_mcell, build_parts(b.max_mcell * Q), Q), kBuildCellsPerBlock * 32, 0, st>>>(
        mol_build_args(s0), reinterpret_cast<const BuildArgs *>(b.tab_molbuild.p));
    g_launches += 6;
}

int batch_nlist_rebuild(Batch &b) {
    const int R = (int)b.reps.size();
    if (!b.tab_grid.p) {
        set_error(MDX_ERR_STATE, "batch tables not built (prepare the batch)");
        return MDX_ERR_STATE;
    }
    const GridArgs *tg = reinterpret_cast<const GridArgs *>(b.tab_grid.p);
    State &s0 = *b.reps[0];
    GridArgs A = grid_args(s0);  // sizing only
    A.n = b.max_n;
    cudaStream_t st = b.stream;
    k_check<<<dim3((b.max_n + 255) / 256, R), 256, 0, st>>>(A, tg, 0);
    MDX_LAUNCHED();
    if (!b.ps.empty()) batch_rebuild_sites(b, st);
    if (!b.mfi.empty()) batch_rebuild_mols(b, st);
    // the per-site replicas' molecule maps (the molecule form's copyback
    // rewrote its own)
    if (!b.ps.empty())
        if (int e = batch_rigid_maps(b)) return e;
    if (s0.e3bFix())
        if (int e = batch_e3b_list(b)) return e;
    if (!b.ps.empty()) {
        GridArgs Ap = A;
        Ap.n = b.max_n_ps;
        k_finish<<<dim3(1, (unsigned)b.ps.size()), 1, 0, st>>>(Ap, reinterpret_cast<const GridArgs *>(b.tab_grid_ps.p));
        MDX_LAUNCHED();
    }
    if (!b.mfi.empty()) {
        GridArgs Am = mol_scan_args(*b.reps[b.mfi[0]]);
        Am.ncell = b.max_mcell;
        k_finish<<<dim3(1, (unsigned)b.mfi.size()), 1, 0, st>>>(Am, reinterpret_cast<const GridArgs *>(b.tab_molscan.p));
        MDX_LAUNCHED();
    }
    MDX_CUDA_TRY(cudaGetLastError());
    return 0;
}

}  // namespace mdx
