// irr_neighbor.cu -- half neighbour list on the GPU by a counting-sort cell list.
//
// Replaces miniMD's serial binned build (miniMD/neighbor.cpp:76-205: linked-list
// bins filled by binatoms :209-239, a half stencil from setup :289-397) and
// moldyn's O(N^2) all-pairs RebuildNeighbor (moldyn/moldyn.cu:552-594):
//   1. each node gets a cell key (cells at least as wide as the list cutoff);
//   2. a stable radix sort by key orders nodes by cell; a count + scan gives
//      each cell's start;
//   3. positions are copied into cell order, so a cell's candidates are
//      contiguous and each is one load, not an id load and then a dependent
//      position load;
//   4. one thread per node (in cell order, so a warp shares cells) scans the
//      27 surrounding cells for partners j > i with r2 <= cut2 and writes them
//      into slots of its own (slot_partners_kernel); warps then sort each row
//      by j and write its pairs (slot_pairs_kernel).  Where the cells do not
//      decide the images, a node has more partners than slots, or the slots do
//      not fit, partners are counted first and written after a scan of the
//      counts (pairs_kernel), then sorted and expanded.  A caller that re-sorts
//      the pairs anyway gets them in no particular order, from a half stencil
//      (pairs_half_kernel: each pair found once, from one end).
// The pair rule is shared bit for bit with the CPU oracle: d = x_i - x_j in
// float, wrapped once by +-box when |d| > box/2 (periodic), r2 = ((dx*dx +
// dy*dy) + dz*dz) with every operation rounded.  Output: pairs (i, j), i < j,
// sorted by i then j -- moldyn's loop order; miniMD lists the same pairs.
// With at least 5 cells per axis and every position inside the periodic box,
// a neighbour cell decides the image of all its partners (list_pair_shifted).
//
// The MD rebuild takes another route (build_rows_by_cell): the nodes are
// re-sorted by the Hilbert index of their cell, and each node's full row is
// written by one search over its 27 cells visited in curve order -- ascending
// by construction, so the rows need neither the pair list, nor atomic row
// cursors, nor a sort.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "irr_internal.cuh"
#include "irr_list_rule.h"
#include "irr_trace.cuh"
#include "../../include/irregular_gb300.h"

namespace irr {
namespace {

struct Grid {
    int nc[3];
    int offs[3][3];   // neighbour cell offsets per axis (deduplicated)
    int noff[3];
    double org[3];
    double inv[3];    // 1 / cell size
    float box, hb, cut2;
    int periodic;
    int fast;         // periodic with >= 5 cells per axis: image decided by the cell
};

__device__ __forceinline__ bool list_pair(float4 a, float4 b, const Grid& g)
{
    float d[3] = {__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)};
    if (g.periodic) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            if (d[c] > g.hb)
                d[c] = __fsub_rn(d[c], g.box);
            else if (d[c] < -g.hb)
                d[c] = __fadd_rn(d[c], g.box);
        }
    }
    const float r2 = __fadd_rn(__fadd_rn(__fmul_rn(d[0], d[0]), __fmul_rn(d[1], d[1])),
                               __fmul_rn(d[2], d[2]));
    return r2 <= g.cut2;
}

// The same rule when the neighbour cell decides the image: with at least 5
// cells per axis and every position in [0, box), a partner in a cell that is
// adjacent without wrapping is less than 2/5 of the box away on that axis
// (the rule keeps d), and one in a cell reached across the boundary more
// than 3/5 (the rule adds or subtracts the box, always the same way), so the
// cell's shift s (0 or +-box) is added instead of compared for.  d + 0 is d
// except for d = -0, whose square is the same.
__device__ __forceinline__ bool list_pair_shifted(float4 a, float4 b, float sx, float sy, float sz,
                                                  float cut2)
{
    const float dx = __fadd_rn(__fsub_rn(a.x, b.x), sx);
    const float dy = __fadd_rn(__fsub_rn(a.y, b.y), sy);
    const float dz = __fadd_rn(__fsub_rn(a.z, b.z), sz);
    const float r2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    return r2 <= cut2;
}

// list_pair_shifted with no shift (a cell reached without crossing the box).
__device__ __forceinline__ bool list_pair_unshifted(float4 a, float4 b, float cut2)
{
    const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
    const float r2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    return r2 <= cut2;
}

template <bool FAST>
__device__ __forceinline__ bool pair_hit(float4 a, float4 b, const Grid& g, float sx, float sy, float sz)
{
    return FAST ? list_pair_shifted(a, b, sx, sy, sz, g.cut2) : list_pair(a, b, g);
}

// Neighbour cell (x, y, z) of a periodic grid wrapped into range, with the
// image shift of each wrapped axis: a cell reached below 0 lies at the top of
// the box (its partners are pulled down by +box), one reached past the top
// at the bottom (-box).
__device__ __forceinline__ void wrap_cell(int& v, int nc, float box, float& s)
{
    s = 0.f;
    if (v < 0) {
        v += nc;
        s = box;
    } else if (v >= nc) {
        v -= nc;
        s = -box;
    }
}

__device__ __forceinline__ int cell_coord(float x, int axis, const Grid& g)
{
    long long k = (long long)floor(((double)x - g.org[axis]) * g.inv[axis]);
    if (g.periodic) k = ((k % g.nc[axis]) + g.nc[axis]) % g.nc[axis];
    if (k < 0) k = 0;
    if (k >= g.nc[axis]) k = g.nc[axis] - 1;
    return (int)k;
}

// Also raises *outside when a position of a periodic box lies outside
// [0, box) (or is NaN): the cell-decided image above then does not hold.
__global__ void cell_keys_kernel(const float4* pos, int64_t n, const __grid_constant__ Grid g, uint32_t* keys,
                                 int32_t* vals, uint32_t* cell_count, int* outside)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float4 p = pos[i];
        if (g.periodic && !(p.x >= 0.f && p.x < g.box && p.y >= 0.f && p.y < g.box && p.z >= 0.f &&
                            p.z < g.box))
            *outside = 1;
        const uint32_t c = ((uint32_t)cell_coord(p.z, 2, g) * g.nc[1] + cell_coord(p.y, 1, g)) *
                               g.nc[0] +
                           cell_coord(p.x, 0, g);
        keys[i] = c;
        vals[i] = (int32_t)i;
        atomicAdd(cell_count + c, 1u);
    }
}

// pos_c[q] = pos[sorted[q]]: positions in cell order, the node's id in w
__global__ void cell_order_kernel(const float4* __restrict__ pos, const int32_t* __restrict__ sorted,
                                  int64_t n, float4* __restrict__ pos_c)
{
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
         q += (int64_t)gridDim.x * blockDim.x)
    {
        const int32_t i = sorted[q];
        float4 p = pos[i];
        p.w = __int_as_float(i);
        pos_c[q] = p;
    }
}

// WRITE == false: counts partners; WRITE == true: writes them from row_off[i],
// as neighbour ids into nbr (with sort_here, sorting the row by j in place:
// only for rows too long for the row sort that otherwise follows) or, when
// pairs != nullptr, as the pairs (i, j) themselves.  FAST: the image decided
// by the cell (list_pair_shifted).
template <bool WRITE, bool FAST>
__device__ __forceinline__ void pairs_rows(const float4* __restrict__ pos_c, const int32_t* __restrict__ sorted,
                                           const uint32_t* __restrict__ cell_start, int64_t n,
                                           const Grid& g, uint32_t* count,
                                           const uint32_t* __restrict__ row_off, int32_t* nbr,
                                           int2* pairs, int sort_here)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int32_t i = sorted[t];
        const float4 a = pos_c[t];
        const int cx = cell_coord(a.x, 0, g), cy = cell_coord(a.y, 1, g), cz = cell_coord(a.z, 2, g);
        uint32_t m = 0;
        const uint32_t base = WRITE ? row_off[i] : 0;
        for (int oz = 0; oz < g.noff[2]; oz++) {
            int z = cz + g.offs[2][oz];
            float sz = 0.f;
            if (FAST) wrap_cell(z, g.nc[2], g.box, sz);
            else if (g.periodic) z = (z + g.nc[2]) % g.nc[2];
            else if (z < 0 || z >= g.nc[2]) continue;
            for (int oy = 0; oy < g.noff[1]; oy++) {
                int y = cy + g.offs[1][oy];
                float sy = 0.f;
                if (FAST) wrap_cell(y, g.nc[1], g.box, sy);
                else if (g.periodic) y = (y + g.nc[1]) % g.nc[1];
                else if (y < 0 || y >= g.nc[1]) continue;
                for (int ox = 0; ox < g.noff[0]; ox++) {
                    int x = cx + g.offs[0][ox];
                    float sx = 0.f;
                    if (FAST) wrap_cell(x, g.nc[0], g.box, sx);
                    else if (g.periodic) x = (x + g.nc[0]) % g.nc[0];
                    else if (x < 0 || x >= g.nc[0]) continue;
                    const uint32_t c = ((uint32_t)z * g.nc[1] + y) * g.nc[0] + x;
                    const uint32_t q1 = cell_start[c + 1];
#pragma unroll 2
                    for (uint32_t q = cell_start[c]; q < q1; q++) {
                        const int32_t j = sorted[q];
                        const float4 b = pos_c[q];
                        if (j <= i) continue;
                        if (pair_hit<FAST>(a, b, g, sx, sy, sz)) {
                            if (WRITE) {
                                if (pairs)
                                    pairs[base + m] = make_int2(i, j);
                                else
                                    nbr[base + m] = j;
                            }
                            m++;
                        }
                    }
                }
            }
        }
        if (!WRITE) {
            count[i] = m;
        } else if (sort_here && !pairs) {
            // insertion sort of the row in place
            for (uint32_t u = 1; u < m; u++) {
                const int32_t v = nbr[base + u];
                uint32_t w = u;
                while (w > 0 && nbr[base + w - 1] > v) {
                    nbr[base + w] = nbr[base + w - 1];
                    w--;
                }
                nbr[base + w] = v;
            }
        }
    }
}

template <bool WRITE>
__global__ void pairs_kernel(const float4* __restrict__ pos_c, const int32_t* __restrict__ sorted,
                             const uint32_t* __restrict__ cell_start, int64_t n,
                             const __grid_constant__ Grid g, const int* __restrict__ outside,
                             uint32_t* count, const uint32_t* __restrict__ row_off, int32_t* nbr,
                             int2* pairs, int sort_here)
{
    if (g.fast && *outside == 0)
        pairs_rows<WRITE, true>(pos_c, sorted, cell_start, n, g, count, row_off, nbr, pairs, sort_here);
    else
        pairs_rows<WRITE, false>(pos_c, sorted, cell_start, n, g, count, row_off, nbr, pairs, sort_here);
}

// The same partners j > i of every node in one pass, into slots of `cap` per
// node (in cell order), where the cell decides the image (open boundaries, or
// Grid::fast and every position in the box; else *over = 1 and nothing is
// written).  cnt[i] = node i's partners; *over is raised when one has more than
// cap.  The cells of a grid row are neighbours in cell order, so a node's 27
// cells are 9 runs of candidates (at the wall of a periodic box up to 18), each
// candidate one 16-byte load that brings its id.
// What bounds it: issue, ~14 instructions a candidate and ~580 candidates a
// node at 64 neighbours.  1,000,003 nodes, list radius 2.8: counting 556 +
// writing 730 us with 27 runs and two loads a candidate -> 474 us.
__global__ void __launch_bounds__(256) slot_partners_kernel(const float4* __restrict__ pos_c,
                                                           const uint32_t* __restrict__ keys,
                                                           const uint32_t* __restrict__ cell_start, int64_t n,
                                                           const __grid_constant__ Grid g,
                                                           const int* __restrict__ outside, uint32_t cap,
                                                           uint32_t* __restrict__ cnt,
                                                           int32_t* __restrict__ slots, int* over)
{
    if (g.periodic && (!g.fast || *outside)) {
        if (threadIdx.x == 0) *over = 1;
        return;
    }
    for (int64_t t0 = (int64_t)blockIdx.x * blockDim.x; t0 < n; t0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = t0 + threadIdx.x;
        if (t >= n) continue;
        const float4 a = pos_c[t];
        const int32_t i = __float_as_int(a.w);
        const uint32_t c = keys[t];
        const int cx = (int)(c % (uint32_t)g.nc[0]), cy = (int)(c / (uint32_t)g.nc[0] % (uint32_t)g.nc[1]),
                  cz = (int)(c / ((uint32_t)g.nc[0] * (uint32_t)g.nc[1]));
        // the block's slots, and the thread's next one and their end in them: 32-bit
        // offsets from one base
        char* const base = reinterpret_cast<char*>(slots + t0 * (int64_t)cap);
        const uint32_t first = threadIdx.x * cap * 4u, end = first + cap * 4u;
        uint32_t at = first;
        auto run = [&](auto shift, uint32_t q, uint32_t q1, float sx, float sy, float sz) {
#pragma unroll 8
            for (; q < q1; q++) {
                const float4 b = pos_c[q];
                const int32_t j = __float_as_int(b.w);
                // no branch: a hit every sixth candidate, so most warps have one
                const bool hit = (j > i) & (decltype(shift)::value ? list_pair_shifted(a, b, sx, sy, sz, g.cut2)
                                                                   : list_pair_unshifted(a, b, g.cut2));
                if (hit & (at < end)) *reinterpret_cast<int32_t*>(base + at) = j;
                at += hit ? 4u : 0u;
            }
        };
        for (int k = 0; k < 9; k++) {
            int z = cz + k / 3 - 1, y = cy + k % 3 - 1;
            float sy = 0.f, sz = 0.f;
            if (g.periodic) {
                wrap_cell(z, g.nc[2], g.box, sz);
                wrap_cell(y, g.nc[1], g.box, sy);
            } else if (z < 0 || z >= g.nc[2] || y < 0 || y >= g.nc[1]) {
                continue;
            }
            const uint32_t row = ((uint32_t)z * g.nc[1] + y) * g.nc[0];
            const int x0 = max(cx - 1, 0), x1 = min(cx + 1, g.nc[0] - 1);
            if (sy == 0.f && sz == 0.f)
                run(std::false_type{}, cell_start[row + x0], cell_start[row + x1 + 1], 0.f, 0.f, 0.f);
            else
                run(std::true_type{}, cell_start[row + x0], cell_start[row + x1 + 1], 0.f, sy, sz);
            if (g.periodic && (cx == 0 || cx == g.nc[0] - 1)) {
                int x = cx == 0 ? -1 : g.nc[0];
                float sx;
                wrap_cell(x, g.nc[0], g.box, sx);
                run(std::true_type{}, cell_start[row + x], cell_start[row + x + 1], sx, sy, sz);
            }
        }
        cnt[i] = (at - first) / 4u;
        if (at > end) *over = 1;
    }
}

// The same pairs from a half stencil, for callers that take the pairs in any
// order (with at least 3 cells per axis, so no cell is its own neighbour):
// node t (in cell order) pairs with the later nodes of its own cell and with
// the nodes of the 13 neighbour cells whose offset (dz, dy, dx) comes after
// (0, 0, 0) in lexicographic order.  Each pair is found once and written as
// (min id, max id).
template <bool WRITE, bool FAST>
__device__ __forceinline__ void half_rows(const float4* __restrict__ pos_c, const int32_t* __restrict__ sorted,
                                          const uint32_t* __restrict__ cell_start, int64_t n,
                                          const Grid& g, uint32_t* count,
                                          const uint32_t* __restrict__ row_off, int2* pairs)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int32_t i = sorted[t];
        const float4 a = pos_c[t];
        const int cx = cell_coord(a.x, 0, g), cy = cell_coord(a.y, 1, g), cz = cell_coord(a.z, 2, g);
        uint32_t m = 0;
        const uint32_t base = WRITE ? row_off[i] : 0;
        for (int o = 0; o < 14; o++) {
            // o = 0: the own cell (later nodes only); o = 1..13: forward offsets
            const int k = o == 0 ? 13 : 13 + o;  // (dz+1)*9 + (dy+1)*3 + (dx+1)
            int z = cz + k / 9 - 1, y = cy + (k / 3) % 3 - 1, x = cx + k % 3 - 1;
            float sx = 0.f, sy = 0.f, sz = 0.f;
            if (g.periodic) {
                wrap_cell(z, g.nc[2], g.box, sz);
                wrap_cell(y, g.nc[1], g.box, sy);
                wrap_cell(x, g.nc[0], g.box, sx);
            } else if (z < 0 || z >= g.nc[2] || y < 0 || y >= g.nc[1] || x < 0 || x >= g.nc[0]) {
                continue;
            }
            const uint32_t c = ((uint32_t)z * g.nc[1] + y) * g.nc[0] + x;
            const uint32_t q1 = cell_start[c + 1];
#pragma unroll 2
            for (uint32_t q = o == 0 ? (uint32_t)t + 1 : cell_start[c]; q < q1; q++) {
                const float4 b = pos_c[q];
                if (pair_hit<FAST>(a, b, g, sx, sy, sz)) {
                    if (WRITE) {
                        const int32_t j = sorted[q];
                        pairs[base + m] = i < j ? make_int2(i, j) : make_int2(j, i);
                    }
                    m++;
                }
            }
        }
        if (!WRITE) count[i] = m;
    }
}

template <bool WRITE>
__global__ void pairs_half_kernel(const float4* __restrict__ pos_c, const int32_t* __restrict__ sorted,
                                  const uint32_t* __restrict__ cell_start, int64_t n,
                                  const __grid_constant__ Grid g, const int* __restrict__ outside,
                                  uint32_t* count, const uint32_t* __restrict__ row_off, int2* pairs)
{
    if (g.fast && *outside == 0)
        half_rows<WRITE, true>(pos_c, sorted, cell_start, n, g, count, row_off, pairs);
    else
        half_rows<WRITE, false>(pos_c, sorted, cell_start, n, g, count, row_off, pairs);
}

// One warp per row: the lanes write consecutive pairs (coalesced stores).
__global__ void expand_pairs_kernel(const uint32_t* row_off, const int32_t* nbr, int64_t n,
                                    int2* edges)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
        const uint32_t k1 = row_off[i + 1];
        for (uint32_t k = row_off[i] + lane; k < k1; k += 32) edges[k] = make_int2((int)i, nbr[k]);
    }
}

// ---- full rows in cell order (the MD rebuild)
// Nodes sorted by the Hilbert index of their cell (cells of the 10-bit curve
// grid: at most 1024 per axis), so each cell's nodes are one contiguous run
// and runs follow the curve; a node's row visits its 27 neighbour cells in
// curve order, so the row comes out ascending with no sort and no atomics.

__device__ __forceinline__ uint32_t cell_of(float4 p, const Grid& g)
{
    return ((uint32_t)cell_coord(p.z, 2, g) * g.nc[1] + cell_coord(p.y, 1, g)) * g.nc[0] +
           cell_coord(p.x, 0, g);
}

// keys[i] = curve index of node i's cell, vals[i] = i; *outside as in cell_keys.
__global__ void cell_curve_keys_kernel(const float4* pos, int64_t n, const __grid_constant__ Grid g,
                                       uint32_t* keys, int32_t* vals, int* outside)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float4 p = pos[i];
        if (g.periodic && !(p.x >= 0.f && p.x < g.box && p.y >= 0.f && p.y < g.box && p.z >= 0.f &&
                            p.z < g.box))
            *outside = 1;
        keys[i] = hilbert10(cell_coord(p.x, 0, g), cell_coord(p.y, 1, g), cell_coord(p.z, 2, g));
        vals[i] = (int32_t)i;
    }
}

// span[c] = [first, end) of cell c's run in the sorted order (0, 0 if empty).
__global__ void cell_spans_kernel(const float4* __restrict__ pos_c, const uint32_t* __restrict__ keys,
                                  int64_t n, const __grid_constant__ Grid g, uint2* span)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t k = keys[t];
        const bool first = t == 0 || keys[t - 1] != k;
        const bool last = t == n - 1 || keys[t + 1] != k;
        if (first || last) {
            const uint32_t c = cell_of(pos_c[t], g);
            if (first) span[c].x = (uint32_t)t;
            if (last) span[c].y = (uint32_t)(t + 1);
        }
    }
}

// Per cell, its 27 neighbour cells (periodic, at least 3 per axis, so all
// distinct) in curve order: {run first, run end, image code}, the code 2 bits
// per axis (1: +box, 2: -box; the shift list_pair_shifted adds) and kOwnCell
// on the cell itself (whose run holds the node: the only one that needs a
// self test).  One warp
// per cell: lane k < 27 takes neighbour k, and a bitonic network over the
// warp's 32 (key, lane) pairs (5 padding keys at the top) puts them in order.
constexpr int kOwnCell = 64;

__global__ void cell_stencil_kernel(const __grid_constant__ Grid g, const uint2* __restrict__ span,
                                    int64_t ncell, int4* table)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < ncell; c += warps) {
        const int cx = (int)(c % g.nc[0]), cy = (int)((c / g.nc[0]) % g.nc[1]),
                  cz = (int)(c / ((int64_t)g.nc[0] * g.nc[1]));
        uint32_t key = 0xffffffffu;
        int4 ent = make_int4(0, 0, 0, 0);
        if (lane < 27) {
            int z = cz + lane / 9 - 1, y = cy + (lane / 3) % 3 - 1, x = cx + lane % 3 - 1;
            float sx, sy, sz;
            wrap_cell(z, g.nc[2], g.box, sz);
            wrap_cell(y, g.nc[1], g.box, sy);
            wrap_cell(x, g.nc[0], g.box, sx);
            const int code = (sx > 0.f ? 1 : sx < 0.f ? 2 : 0) | (sy > 0.f ? 4 : sy < 0.f ? 8 : 0) |
                             (sz > 0.f ? 16 : sz < 0.f ? 32 : 0) | (lane == 13 ? kOwnCell : 0);
            const uint2 sp = span[((int64_t)z * g.nc[1] + y) * g.nc[0] + x];
            key = hilbert10((uint32_t)x, (uint32_t)y, (uint32_t)z);
            ent = make_int4((int)sp.x, (int)sp.y, code, 0);
        }
        int src = lane;  // whose entry this lane holds after the network
#pragma unroll
        for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                const uint32_t ok = __shfl_xor_sync(0xffffffffu, key, stride);
                const int os = __shfl_xor_sync(0xffffffffu, src, stride);
                const bool up = (lane & size) == 0;
                const bool lower = (lane & stride) == 0;
                // keep the smaller key in the lower lane of an ascending pair
                const bool take = (up == lower) ? (ok < key) : (ok > key);
                if (take) {
                    key = ok;
                    src = os;
                }
            }
        }
        const int4 got = make_int4(__shfl_sync(0xffffffffu, ent.x, src), __shfl_sync(0xffffffffu, ent.y, src),
                                   __shfl_sync(0xffffffffu, ent.z, src), 0);
        if (lane < 27) table[c * 27 + lane] = got;
    }
}

__device__ __forceinline__ float image_shift(int code, float box)
{
    return code == 1 ? box : (code == 2 ? -box : 0.f);
}

// MODE kCount: deg[t] = row length.  kWrite: the row's columns from
// row_off[t], ascending.  kScratch: both in one pass, the columns into a
// fixed-capacity slot scratch[t * cap, +cap) (the count goes on past cap, so
// an overflowing row is known and its entries are not stored).  864,000 atoms,
// list radius 2.8, ~500 candidates and 78 partners each: one pass 550 us with a
// branch per hit and 64-bit addresses, 475 without.  What bounds it: issue, and
// the scattered 4-byte writes (counting alone takes 360).
enum RowsMode { kCount = 0, kWrite = 1, kScratch = 2 };

template <int MODE, bool FAST>
__device__ __forceinline__ void cell_rows_body(const float4* __restrict__ pos_c, int64_t n, const Grid& g,
                                               const int4* __restrict__ table, uint32_t* deg,
                                               const uint32_t* __restrict__ row_off, int32_t* col,
                                               uint32_t cap)
{
    for (int64_t t0 = (int64_t)blockIdx.x * blockDim.x; t0 < n; t0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = t0 + threadIdx.x;
        if (t >= n) continue;
        const float4 a = pos_c[t];
        const int4* st = table + (int64_t)cell_of(a, g) * 27;
        // bytes: the row's next entry and, of slots, their end, from one base for
        // the block (a row written in place has its own)
        char* const base = reinterpret_cast<char*>(MODE == kWrite ? col + row_off[t]
                                                   : MODE == kScratch ? col + t0 * (int64_t)cap : nullptr);
        const uint32_t first = MODE == kScratch ? threadIdx.x * cap * 4u : 0u, end = first + cap * 4u;
        uint32_t at = first;
        // one run of candidates; SELF: the node's own run (skip q == t),
        // SHIFT: a run across the box boundary (FAST only: elsewhere the cell
        // decides no shift, and the rule's own test runs when !FAST)
        auto run = [&](auto self, auto shift, uint32_t q, uint32_t q1, float sx, float sy, float sz) {
            constexpr bool SELF = decltype(self)::value, SHIFT = decltype(shift)::value;
#pragma unroll 8
            for (; q < q1; q++) {
                const float4 b = pos_c[q];
                bool hit;
                if (!FAST)
                    hit = list_pair(a, b, g);
                else if (SHIFT)
                    hit = list_pair_shifted(a, b, sx, sy, sz, g.cut2);
                else
                    hit = list_pair_unshifted(a, b, g.cut2);
                if (SELF) hit = hit & (q != (uint32_t)t);
                // no branch: most warps have a hit
                if (MODE != kCount && (hit & (MODE == kWrite || at < end)))
                    *reinterpret_cast<int32_t*>(base + at) = (int32_t)q;
                at += hit ? 4u : 0u;
            }
        };
        using T = std::true_type;
        using F = std::false_type;
        for (int k = 0; k < 27; k++) {
            const int4 e = st[k];
            const uint32_t q0 = (uint32_t)e.x, q1 = (uint32_t)e.y;
            if (e.z & kOwnCell) {
                run(T{}, F{}, q0, q1, 0.f, 0.f, 0.f);
            } else if (FAST && e.z != 0) {
                run(F{}, T{}, q0, q1, image_shift(e.z & 3, g.box), image_shift((e.z >> 2) & 3, g.box),
                    image_shift((e.z >> 4) & 3, g.box));
            } else {
                run(F{}, F{}, q0, q1, 0.f, 0.f, 0.f);
            }
        }
        if (MODE != kWrite) deg[t] = (at - first) / 4u;
    }
}

// The same with L lanes per node: a run's candidates L at a time, the hits of
// a step placed by a ballot, so in the same order.
template <int MODE, bool FAST, int L>
__device__ __forceinline__ void cell_rows_lanes(const float4* __restrict__ pos_c, int64_t n, const Grid& g,
                                                const int4* __restrict__ table, uint32_t* deg,
                                                const uint32_t* __restrict__ row_off, int32_t* col, uint32_t cap)
{
    const int lane = threadIdx.x & 31, l = lane % L, first = lane - l;
    const int64_t stride = (((int64_t)gridDim.x * blockDim.x) >> 5) * (32 / L);
    for (int64_t t0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (32 / L); t0 < n; t0 += stride) {
        const bool is = t0 + lane / L < n;
        const int64_t t = is ? t0 + lane / L : n - 1;
        const float4 a = pos_c[t];
        const int4* st = table + (int64_t)cell_of(a, g) * 27;
        int32_t* out = MODE == kWrite ? col + row_off[t] : (MODE == kScratch ? col + t * (int64_t)cap : nullptr);
        uint32_t m = 0;
        int4 e = st[0];
        for (int k = 0; k < 27; k++) {
            const int4 next = st[k < 26 ? k + 1 : k];
            const int count = is ? e.y - e.x : 0;
            const int most = __reduce_max_sync(0xffffffffu, count);
            const float sx = image_shift(e.z & 3, g.box), sy = image_shift((e.z >> 2) & 3, g.box),
                        sz = image_shift((e.z >> 4) & 3, g.box);
            for (int x0 = 0; x0 < most; x0 += 4 * L) {  // 4 of a lane's candidates in flight
                float4 b[4];
#pragma unroll
                for (int y = 0; y < 4; y++) {
                    const int x = x0 + y * L + l;
                    b[y] = pos_c[x < count ? (int64_t)e.x + x : t];
                }
#pragma unroll
                for (int y = 0; y < 4; y++) {
                    if (x0 + y * L >= most) break;
                    const int x = x0 + y * L + l;
                    const int64_t q = x < count ? (int64_t)e.x + x : t;
                    const bool hit = pair_hit<FAST>(a, b[y], g, sx, sy, sz) && q != t;
                    const uint32_t hits = (__ballot_sync(0xffffffffu, hit) >> first) & ((1u << L) - 1u);
                    const uint32_t at = m + (uint32_t)__popc(hits & ((1u << l) - 1u));
                    if (MODE != kCount && hit && (MODE == kWrite || at < cap)) out[at] = (int32_t)q;
                    m += (uint32_t)__popc(hits);
                }
            }
            e = next;
        }
        if (MODE != kWrite && is && l == 0) deg[t] = m;
    }
}

// Scratch rows (cap apart) packed into col at row_off: one warp per row.
__global__ void compact_rows_kernel(const int32_t* __restrict__ scratch, uint32_t cap,
                                    const uint32_t* __restrict__ row_off, int64_t n, int32_t* __restrict__ col)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < n; t += warps) {
        const uint32_t b = row_off[t], len = row_off[t + 1] - b;
        const int32_t* src = scratch + t * (int64_t)cap;
        for (uint32_t k = lane; k < len; k += 32) col[b + k] = src[k];
    }
}

// total[0] += sum of deg[0, n) in 64 bits (the row offsets are 32-bit: the
// caller refuses a list whose entries do not fit), and total[1] = max(total[1], the longest row).
__global__ void sum_u32_kernel(const uint32_t* __restrict__ deg, int64_t n, unsigned long long* total)
{
    unsigned long long w = 0, mx = 0;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x) {
        w += deg[t];
        mx = deg[t] > mx ? deg[t] : mx;
    }
    for (int off = 16; off > 0; off >>= 1) {
        w += __shfl_down_sync(0xffffffffu, w, off);
        const unsigned long long o = __shfl_down_sync(0xffffffffu, mx, off);
        mx = o > mx ? o : mx;
    }
    if ((threadIdx.x & 31) == 0) {
        if (w) atomicAdd(total, w);
        if (mx) atomicMax(total + 1, mx);
    }
}

template <int MODE, int L>
__global__ void cell_rows_kernel(const float4* __restrict__ pos_c, int64_t n, const __grid_constant__ Grid g,
                                 const int* __restrict__ outside, const int4* __restrict__ table,
                                 uint32_t* deg, const uint32_t* __restrict__ row_off, int32_t* col,
                                 uint32_t cap)
{
    const bool fast = g.fast && *outside == 0;
    if constexpr (L > 1) {
        if (fast) cell_rows_lanes<MODE, true, L>(pos_c, n, g, table, deg, row_off, col, cap);
        else cell_rows_lanes<MODE, false, L>(pos_c, n, g, table, deg, row_off, col, cap);
    } else {
        if (fast) cell_rows_body<MODE, true>(pos_c, n, g, table, deg, row_off, col, cap);
        else cell_rows_body<MODE, false>(pos_c, n, g, table, deg, row_off, col, cap);
    }
}

int grid_of(int64_t n)
{
    int64_t g = (n + 255) / 256;
    return (int)(g < 1 ? 1 : (g > 8192 ? 8192 : g));
}

}  // namespace

namespace {

// The cell grid of a list cutoff: cells at least as wide as the cutoff (so a
// partner is in the same or an adjacent cell), at most 1024 per axis and a
// few per node; a periodic axis of fewer than 3 cells becomes one cell.
cudaError_t make_grid(const float4* pos, int64_t n, float box, float cut2, Grid* out, cudaStream_t s)
{
    Grid g{};
    g.periodic = box > 0.0f;
    g.box = box;
    g.hb = 0.5f * box;
    g.cut2 = cut2;
    const double cut = std::sqrt((double)cut2) * 1.0001 + 1e-12;
    double lo[3] = {0, 0, 0}, ext[3] = {box, box, box};
    if (!g.periodic) {
        float flo[3], fhi[3];
        IRR_CUDA_TRY(bbox_minmax(pos, n, flo, fhi, s));
        for (int c = 0; c < 3; c++) {
            lo[c] = flo[c];
            ext[c] = (double)fhi[c] - (double)flo[c];
        }
    }
    for (int c = 0; c < 3; c++) {
        int k = (int)std::floor(ext[c] / cut);
        if (g.periodic && k < 3) k = 1;
        if (k < 1) k = 1;
        if (k > 1024) k = 1024;
        g.nc[c] = k;
    }
    // keep the cell count within a few cells per node (coarser cells stay valid)
    while ((double)g.nc[0] * g.nc[1] * g.nc[2] > 8.0 * (double)n + 64.0) {
        int a = (g.nc[0] >= g.nc[1] && g.nc[0] >= g.nc[2]) ? 0 : (g.nc[1] >= g.nc[2] ? 1 : 2);
        g.nc[a] = g.nc[a] / 2;
        if (g.periodic && g.nc[a] < 3) g.nc[a] = 1;
        if (g.nc[a] < 1) g.nc[a] = 1;
    }
    for (int c = 0; c < 3; c++) {
        g.org[c] = g.periodic ? 0.0 : lo[c];
        // slightly wider cells than ext/nc so the max coordinate maps inside
        // (clamped anyway); the layout never decides a pair, the rule does
        const double csz = ext[c] > 0 ? ext[c] / g.nc[c] : 1.0;
        g.inv[c] = 1.0 / csz;
        if (g.nc[c] >= 3) {
            g.offs[c][0] = -1; g.offs[c][1] = 0; g.offs[c][2] = 1; g.noff[c] = 3;
        } else if (g.nc[c] == 2) {
            g.offs[c][0] = 0; g.offs[c][1] = 1; g.noff[c] = 2;
            if (!g.periodic) { g.offs[c][0] = -1; g.offs[c][1] = 0; g.offs[c][2] = 1; g.noff[c] = 3; }
        } else {
            g.offs[c][0] = 0; g.noff[c] = 1;
        }
    }
    g.fast = g.periodic && g.nc[0] >= 5 && g.nc[1] >= 5 && g.nc[2] >= 5;
    *out = g;
    return cudaSuccess;
}

}  // namespace

namespace {

// One search pass into slots of cap per node, then the list from them.  *done is
// false where the slots do not do (no room for them or for the list beside
// them, a node of more than cap partners, cells that do not decide the images):
// the caller then counts first.  aux: 2 words.
cudaError_t list_by_slots(const float4* pos_c, const uint32_t* keys, const int32_t* sorted, const uint32_t* cell_start,
                          int64_t n, const Grid& g, const int* outside, uint32_t cap, uint32_t* cnt, uint32_t* aux,
                          int2** d_edges, int64_t* num_edges, bool* done, cudaStream_t s)
{
    *done = false;
    Temps tmp{s, {}};
    int32_t* slots = nullptr;
    cudaError_t e = tmp.get(&slots, (size_t)cap * (size_t)n);
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();
    if (e != cudaSuccess) return e == cudaErrorMemoryAllocation ? cudaSuccess : e;
    IRR_CUDA_TRY(cudaMemsetAsync(aux, 0, 2 * sizeof(uint32_t), s));
    slot_partners_kernel<<<grid_of(n), 256, 0, s>>>(pos_c, keys, cell_start, n, g, outside, cap, cnt, slots,
                                                    reinterpret_cast<int*>(aux + 1));
    IRR_CUDA_TRY(cudaGetLastError());
    IRR_CUDA_TRY(cudaMemsetAsync(cnt + n, 0, sizeof(uint32_t), s));
    IRR_CUDA_TRY(scan_exclusive_u32(cnt, cnt, n + 1, aux, s));
    uint32_t got[2] = {0, 0};
    IRR_CUDA_TRY(cudaMemcpyAsync(got, aux, sizeof(got), cudaMemcpyDeviceToHost, s));
    IRR_CUDA_TRY(cudaStreamSynchronize(s));
    if (got[1] || got[0] > 0x7fffffffu) return cudaSuccess;
    if (got[0] > 0) {
        int2* edges = nullptr;
        e = irr_malloc_list((void**)&edges, sizeof(int2) * got[0]);
        if (e == cudaErrorMemoryAllocation) cudaGetLastError();
        if (e != cudaSuccess) return e == cudaErrorMemoryAllocation ? cudaSuccess : e;
        e = launch_slot_pairs(cnt, sorted, n, slots, cap, edges, s);
        if (e != cudaSuccess) {
            irr_free_list(edges);
            return e;
        }
        *d_edges = edges;
    }
    *num_edges = got[0];
    *done = true;
    return cudaSuccess;
}

}  // namespace

cudaError_t build_neighbor_list(const float4* pos, int64_t n, float box, float cut2,
                                int2** d_edges, int64_t* num_edges, cudaStream_t s, bool sort_rows)
{
    *d_edges = nullptr;
    *num_edges = 0;
    if (n <= 1) return cudaSuccess;
    Grid g{};
    IRR_CUDA_TRY(make_grid(pos, n, box, cut2, &g, s));
    const int64_t ncell = (int64_t)g.nc[0] * g.nc[1] * g.nc[2];
    Temps tmp{s, {}};
    uint32_t *keys = nullptr, *keys_tmp = nullptr, *cell_start = nullptr, *cnt = nullptr;
    int32_t *sorted = nullptr, *vals_tmp = nullptr;
    float4* pos_c = nullptr;
    IRR_CUDA_TRY(tmp.get(&keys, n));
    IRR_CUDA_TRY(tmp.get(&keys_tmp, n));
    IRR_CUDA_TRY(tmp.get(&sorted, n));
    IRR_CUDA_TRY(tmp.get(&vals_tmp, n));
    IRR_CUDA_TRY(tmp.get(&cell_start, ncell + 1));
    // cnt[n + 1]: the flag that some position lies outside the box
    IRR_CUDA_TRY(tmp.get(&cnt, n + 2));
    int* outside = reinterpret_cast<int*>(cnt + n + 1);
    IRR_CUDA_TRY(cudaMemsetAsync(cell_start, 0, sizeof(uint32_t) * (ncell + 1), s));
    IRR_CUDA_TRY(cudaMemsetAsync(outside, 0, sizeof(int), s));
    cell_keys_kernel<<<grid_of(n), 256, 0, s>>>(pos, n, g, keys, sorted, cell_start, outside);
    IRR_CUDA_TRY(cudaGetLastError());
    int bits = 1;
    while (bits < 32 && ((int64_t)1 << bits) < ncell) bits++;
    IRR_CUDA_TRY(radix_sort_pairs(keys, sorted, keys_tmp, vals_tmp, n, bits, s));
    IRR_CUDA_TRY(scan_exclusive_u32(cell_start, cell_start, ncell + 1, nullptr, s));
    IRR_CUDA_TRY(tmp.get(&pos_c, n));
    cell_order_kernel<<<grid_of(n), 256, 0, s>>>(pos, sorted, n, pos_c);
    IRR_CUDA_TRY(cudaGetLastError());
    // rows in order: one search pass into slots, where the cells decide the images
    double volume = 1.0;
    for (int c = 0; c < 3; c++) volume *= g.periodic ? (double)box : std::max(g.nc[c] / g.inv[c], std::sqrt((double)cut2));
    const double sphere = volume > 0 ? 4.18879 * cut2 * std::sqrt((double)cut2) * n / volume : (double)n;
    const uint32_t cap = sort_rows && (g.fast || !g.periodic) ? list_slots(sphere, n, kRowSortMax) : 0u;
    if (cap > 0) {
        bool done = false;
        IRR_CUDA_TRY(list_by_slots(pos_c, keys, sorted, cell_start, n, g, outside, cap, cnt, keys_tmp, d_edges,
                                   num_edges, &done, s));
        if (done) return cudaSuccess;
    }
    // rows in any order are asked for: the half stencil, where the box allows it
    const bool half = !sort_rows && g.nc[0] >= 3 && g.nc[1] >= 3 && g.nc[2] >= 3;
    if (half)
        pairs_half_kernel<false><<<grid_of(n), 256, 0, s>>>(pos_c, sorted, cell_start, n, g, outside,
                                                            cnt, nullptr, nullptr);
    else
        pairs_kernel<false><<<grid_of(n), 256, 0, s>>>(pos_c, sorted, cell_start, n, g, outside, cnt,
                                                       nullptr, nullptr, nullptr, 0);
    IRR_CUDA_TRY(cudaGetLastError());
    IRR_CUDA_TRY(cudaMemsetAsync(cnt + n, 0, sizeof(uint32_t), s));
    uint32_t* d_total = keys_tmp;  // reuse as the total's slot
    IRR_CUDA_TRY(scan_exclusive_u32(cnt, cnt, n + 1, d_total, s));
    uint32_t total = 0;
    IRR_CUDA_TRY(cudaMemcpyAsync(&total, d_total, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    IRR_CUDA_TRY(cudaStreamSynchronize(s));
    if ((int64_t)total > 0x7fffffffLL) return cudaErrorInvalidValue;
    if (total == 0) return cudaSuccess;
    int2* edges = nullptr;
    IRR_CUDA_TRY(sort_rows ? irr_malloc_list((void**)&edges, sizeof(int2) * total)
                           : irr_malloc_async((void**)&edges, sizeof(int2) * total, s));
    auto write = [&]() -> cudaError_t {
        if (sort_rows) {
            uint32_t longest = 0;
            IRR_CUDA_TRY(max_row_len(cnt, n, &longest, s));
            const int sort_here = longest > (uint32_t)kRowSortMax;
            int32_t* nbr = nullptr;
            IRR_CUDA_TRY(tmp.get(&nbr, total));
            pairs_kernel<true><<<grid_of(n), 256, 0, s>>>(pos_c, sorted, cell_start, n, g, outside,
                                                          nullptr, cnt, nbr, nullptr, sort_here);
            IRR_CUDA_TRY(cudaGetLastError());
            if (!sort_here) IRR_CUDA_TRY(launch_row_sort(cnt, n, nbr, s));
            expand_pairs_kernel<<<grid_of(32 * n), 256, 0, s>>>(cnt, nbr, n, edges);
        } else if (half) {
            pairs_half_kernel<true><<<grid_of(n), 256, 0, s>>>(pos_c, sorted, cell_start, n, g,
                                                               outside, nullptr, cnt, edges);
        } else {
            pairs_kernel<true><<<grid_of(n), 256, 0, s>>>(pos_c, sorted, cell_start, n, g, outside,
                                                          nullptr, cnt, nullptr, edges, 0);
        }
        return cudaGetLastError();
    };
    const cudaError_t e = write();
    if (e != cudaSuccess) {
        if (sort_rows) {
            cudaStreamSynchronize(s);
            irr_free_list(edges);
        } else {
            cudaFreeAsync(edges, s);
        }
        return e;
    }
    *d_edges = edges;
    *num_edges = total;
    return cudaSuccess;
}

namespace {

// Where the nodes are too few warps to hide the search's latency, 8 lanes share
// a node's candidates.  100 MD steps with 5 rebuilds, us with 8 lanes a node and
// with one: 6,912 nodes 1980 and 2195, 16,384 2274 and 2497, 32,000 2513 and 2602,
// 37,044 2966 and 3028, 42,592 3163 and 3131, 55,296 3329 and 3256, 70,304 3907 and
// 3728.
constexpr int64_t kLanesNodes = 40000;

template <int MODE>
void launch_cell_rows(const float4* pos_c, int64_t n, const Grid& g, const int* outside, const int4* table,
                      uint32_t* deg, const uint32_t* row_off, int32_t* col, uint32_t cap, cudaStream_t s)
{
    if (n <= kLanesNodes)
        cell_rows_kernel<MODE, 8><<<grid_of(8 * n), 256, 0, s>>>(pos_c, n, g, outside, table, deg, row_off, col, cap);
    else
        cell_rows_kernel<MODE, 1><<<grid_of(n), 256, 0, s>>>(pos_c, n, g, outside, table, deg, row_off, col, cap);
}

}  // namespace

cudaError_t build_rows_by_cell(const float4* pos, int64_t n, float box, float cut2, PartitionOut* out,
                               int64_t* num_edges, uint32_t* longest, uint32_t cap_hint, cudaStream_t s)
{
    *out = PartitionOut{};
    *num_edges = 0;
    *longest = 0;
    if (n <= 1 || !(box > 0.0f) || n > 0x7fffffffLL) return cudaErrorNotSupported;
    Grid g{};
    IRR_CUDA_TRY(make_grid(pos, n, box, cut2, &g, s));  // periodic: host arithmetic only
    const int64_t ncell = (int64_t)g.nc[0] * g.nc[1] * g.nc[2];
    if (g.nc[0] < 3 || g.nc[1] < 3 || g.nc[2] < 3 || ncell > n) return cudaErrorNotSupported;
    Temps tmp{s, {}};
    uint32_t *keys = nullptr, *keys_tmp = nullptr;
    int32_t* vals_tmp = nullptr;
    float4* pos_c = nullptr;
    uint2* span = nullptr;
    int4* table = nullptr;
    unsigned long long* aux = nullptr;  // [0] the entry count, [1] the longest row, [2] the outside flag
    PartitionOut p;
    auto run = [&]() -> cudaError_t {
        IRR_CUDA_TRY(irr_malloc_async((void**)&p.perm, sizeof(int32_t) * n, s));
        IRR_CUDA_TRY(irr_malloc_async((void**)&p.row_off, sizeof(uint32_t) * (n + 1), s));
        IRR_CUDA_TRY(tmp.get(&keys, n));
        IRR_CUDA_TRY(tmp.get(&keys_tmp, n));
        IRR_CUDA_TRY(tmp.get(&vals_tmp, n));
        IRR_CUDA_TRY(tmp.get(&pos_c, n));
        IRR_CUDA_TRY(tmp.get(&span, ncell));
        IRR_CUDA_TRY(tmp.get(&table, ncell * 27));
        IRR_CUDA_TRY(tmp.get(&aux, 3));
        // one search pass into cap_hint slots per node when they fit in memory;
        // otherwise (and at the first build) a counting pass, then the writing one
        bool one_pass = false;
        if (cap_hint > 0 && cap_hint <= 4096) {
            one_pass = irr_malloc_async((void**)&p.slots, sizeof(int32_t) * (size_t)n * cap_hint, s) == cudaSuccess;
            p.cap = cap_hint;
            if (!one_pass) {
                cudaGetLastError();
                p.slots = nullptr;
            }
        }
        IRR_CUDA_TRY(cudaMemsetAsync(span, 0, sizeof(uint2) * ncell, s));
        IRR_CUDA_TRY(cudaMemsetAsync(aux, 0, 3 * sizeof(unsigned long long), s));
        int* outside = reinterpret_cast<int*>(aux + 2);
        const int gn = grid_of(n);
        cell_curve_keys_kernel<<<gn, 256, 0, s>>>(pos, n, g, keys, p.perm, outside);
        IRR_CUDA_TRY(cudaGetLastError());
        // coordinates below 2^b give curve indices below 8^b: the levels above
        // only exchange axes
        int bits = 0;
        while ((1 << bits) < std::max(g.nc[0], std::max(g.nc[1], g.nc[2]))) bits++;
        IRR_CUDA_TRY(radix_sort_pairs(keys, p.perm, keys_tmp, vals_tmp, n, 3 * bits, s));
        cell_order_kernel<<<gn, 256, 0, s>>>(pos, p.perm, n, pos_c);
        cell_spans_kernel<<<gn, 256, 0, s>>>(pos_c, keys, n, g, span);
        cell_stencil_kernel<<<grid_of(32 * ncell), 256, 0, s>>>(g, span, ncell, table);
        if (one_pass)
            launch_cell_rows<kScratch>(pos_c, n, g, outside, table, p.row_off, nullptr, p.slots, cap_hint, s);
        else
            launch_cell_rows<kCount>(pos_c, n, g, outside, table, p.row_off, nullptr, nullptr, 0, s);
        sum_u32_kernel<<<gn < 256 ? gn : 256, 256, 0, s>>>(p.row_off, n, aux);  // few atomics
        IRR_CUDA_TRY(cudaGetLastError());
        unsigned long long host_aux[2] = {0, 0};
        IRR_CUDA_TRY(cudaMemcpyAsync(host_aux, aux, sizeof(host_aux), cudaMemcpyDeviceToHost, s));
        IRR_CUDA_TRY(cudaStreamSynchronize(s));
        const unsigned long long total = host_aux[0];
        if (total > 0x7fffffffull) return cudaErrorInvalidValue;
        IRR_CUDA_TRY(cudaMemsetAsync(p.row_off + n, 0, sizeof(uint32_t), s));
        IRR_CUDA_TRY(scan_exclusive_u32(p.row_off, p.row_off, n + 1, nullptr, s));
        if (!one_pass || host_aux[1] > cap_hint) {
            // a row longer than the slots (or no scratch): search again, writing in place
            if (p.slots) cudaFreeAsync(p.slots, s);
            p.slots = nullptr;
            IRR_CUDA_TRY(alloc_col(&p.col, (int64_t)total, s));
            launch_cell_rows<kWrite>(pos_c, n, g, outside, table, nullptr, p.row_off, p.col, 0, s);
        }
        IRR_CUDA_TRY(cudaGetLastError());
        *num_edges = (int64_t)(total / 2);
        *longest = (uint32_t)host_aux[1];
        return cudaSuccess;
    };
    const cudaError_t e = run();
    if (e != cudaSuccess) {
        if (p.perm) cudaFreeAsync(p.perm, s);
        if (p.row_off) cudaFreeAsync(p.row_off, s);
        if (p.col) cudaFreeAsync(p.col, s);
        if (p.slots) cudaFreeAsync(p.slots, s);
        *num_edges = 0;
        *longest = 0;
        return e;
    }
    *out = p;
    return cudaSuccess;
}

cudaError_t pack_rows(PartitionOut* p, int64_t n, int64_t m, cudaStream_t s)
{
    if (!p->slots) return cudaSuccess;
    IRR_CUDA_TRY(alloc_col(&p->col, m, s));
    compact_rows_kernel<<<grid_of(32 * n), 256, 0, s>>>(p->slots, (uint32_t)p->cap, p->row_off, n, p->col);
    return cudaGetLastError();
}

}  // namespace irr

extern "C" {

int irr_neighbor_build(int device, void* stream, const void* pos, int pos_elm, int pos_on_device,
                       int64_t n, float box, float list_cut2, int32_t** d_edges,
                       int64_t* num_edges)
{
    irr::TraceRange trace_("irr_neighbor_build");
    if (!d_edges || !num_edges || n < 0 || (n > 0 && !pos)) return IRR_ERR_ARG;
    if (pos_elm != 12 && pos_elm != 16 && pos_elm != 24) return IRR_ERR_ARG;
    if (!(box >= 0.0f) || !(list_cut2 >= 0.0f) || !std::isfinite(box) || !std::isfinite(list_cut2))
        return IRR_ERR_ARG;
    if (n > 0x7fffffffLL) return IRR_ERR_CAPACITY;
    *d_edges = nullptr;
    *num_edges = 0;
    irr::DeviceGuard dev_guard(device);
    if (!dev_guard.ok()) return IRR_ERR_CUDA;
    cudaStream_t s = (cudaStream_t)stream;
    void* raw = nullptr;
    float4* p4 = nullptr;
    int rc = IRR_OK;
    cudaError_t e = cudaSuccess;
    const void* src = pos;
    if (n > 0 && !pos_on_device) {
        e = irr::irr_malloc_async(&raw, (size_t)n * pos_elm, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(raw, pos, (size_t)n * pos_elm, cudaMemcpyHostToDevice, s);
        src = raw;
    }
    if (e == cudaSuccess && n > 0) e = irr::irr_malloc_async(&p4, sizeof(float4) * (size_t)n, s);
    if (e == cudaSuccess && n > 0) e = irr::launch_load_nodes(src, pos_elm, nullptr, n, p4, s);
    int2* edges = nullptr;
    int64_t cnt = 0;
    if (e == cudaSuccess) e = irr::build_neighbor_list(p4, n, box, list_cut2, &edges, &cnt, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        rc = (e == cudaErrorMemoryAllocation) ? IRR_ERR_NOMEM : (e == cudaErrorInvalidValue ? IRR_ERR_CAPACITY : IRR_ERR_CUDA);
        if (edges) {
            cudaStreamSynchronize(s);
            irr::irr_free_list(edges);
        }
        edges = nullptr;
        cnt = 0;
    }
    if (raw) cudaFreeAsync(raw, s);
    if (p4) cudaFreeAsync(p4, s);
    *d_edges = (int32_t*)edges;
    *num_edges = cnt;
    return rc;
}

int irr_device_free(int device, void* d_ptr)
{
    if (!d_ptr) return IRR_OK;
    irr::DeviceGuard dev_guard(device);
    if (!dev_guard.ok() || cudaDeviceSynchronize() != cudaSuccess || irr::irr_free_list(d_ptr) != cudaSuccess) {
        cudaGetLastError();
        return IRR_ERR_CUDA;
    }
    irr::irr_pool_trim(device);
    return IRR_OK;
}

}  // extern "C"
