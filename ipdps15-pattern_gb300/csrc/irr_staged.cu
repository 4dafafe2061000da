// irr_staged.cu -- the staged ("halo") entry layout, built on the GPU.
//
// The partitioned reduction gathers every neighbour's position for every
// directed entry.  In the sliced layout those gathers go through L1 and, for
// ~15 % of the lines, to L2: the kernel waits on them and the L1 data pipe
// does ~9.5 wavefronts per 32-lane gather.  Here each work item (a run of up
// to 8 slices of 8 consecutive curve-ordered rows) carries its own table: the
// sorted distinct ids of its rows and of all their neighbours -- ~465 for 64
// rows at ~64 neighbours each, so every staged position is used ~9 times.
// The kernel's producer warp gathers the table's positions into shared memory
// (cp.async) while the consumers work on the item before; the consumers then
// read positions from shared memory by 16-bit table offsets.  A row's entries
// are ordered so that the 8 lanes of each quarter-warp phase of a 128-bit
// shared load mostly hit 8 different bank groups: row i of a slice takes its
// pick (t, h, l) from bank group (2t + h + 4 (i & 1) + l) mod 8 -- the rows of
// a phase take complementary groups, and the window rotates so that a row
// draws on all 8 groups evenly -- else from its fullest group.  On a curve-
// ordered random box at ~64 neighbours that is ~5.4 wavefronts per 128-bit
// gather (8 lanes at random would be ~7.2 with the table sorted, ~9 unsorted).
//
// Layout (the oracle restates it bit for bit, oracle/irr_oracle.c
// orc_staged_layout):
//   items: blocks of 8 consecutive rows, cut into runs of at most
//   kHaloSlicesPerItem blocks and `stream` words (a block counted at
//   its longest row), each run cut into the longest prefixes whose table
//   holds at most `tab` ids;
//   slices: within an item the rows are ordered longest first (ties by row),
//   and slice j takes rows 8j .. 8j + 7 of that order -- rows of similar
//   length, so a slice pads ~8 % instead of ~17 % for 8 consecutive rows (the
//   table, and so every gather, is the item's whatever the order); slice j
//   takes 32 (T_j + 1) words, T_j = ceil(its longest row / 8): a header word
//   own | len << 14 | lrow << 24 per lane (own: the row's byte offset in the
//   table, lrow: its index in the item; 1 << 31 for a padding row), then one
//   word b0 | b1 << 16 per lane and step -- 16-bit byte offsets into the
//   table of the lane's two entries (padding: the row's own offset).
// Build, all on the device (the host learns the sizes, nothing else):
//   block_runs_kernel  the longest run starting at each block, and each tile's
//                      map from the block a run enters it at to the next tile's;
//   run_entries_kernel the entries of a greedy cut from block 0, by composing
//   list_runs_kernel   those maps (8 states), and its runs;
//   cut_runs_kernel    one CTA per run: the items' tables counted, their words;
//   place_items_kernel the items' places in the words and tables;
//   fill_items_kernel  one CTA per item: its table, words and slice offsets.
// A table is gathered as a hash of 32-id groups with a bit per id: neighbours
// on the curve share groups, so ~465 ids are ~120 groups to sort, and an id's
// slot is its group's first slot plus a population count -- no search.
// What bounds it: instruction issue (a hash probe and a bucket per entry).
// 1,000,003 nodes at 64 neighbours: counting 228 -> 173 us, filling 1129 -> 722 us,
// and the cut, the row offsets' copy to the host and the per-run counts' copies
// (~1.6 ms on the host) are gone.
#include <algorithm>
#include <climits>
#include <vector>

#include "irr_internal.cuh"

namespace irr {
namespace {

constexpr int kPick = 8;                         // slices of an item, blocks of a run: at most
// The limits of the two variants.
struct NarrowItem {
    static constexpr int kTab = kHaloTabMax, kStream = kHaloStreamMax;
    static constexpr int kHash = 1024, kThreads = 128, kCtas = 7, kHeld = 4, kCutAhead = 2;
};
struct WideItem {
    static constexpr int kTab = kHaloWideTabMax, kStream = kHaloWideStreamMax;
    static constexpr int kHash = 2048, kThreads = 256, kCtas = 3, kHeld = 8, kCutAhead = 4;
};
static_assert(kHaloTabMax < 1024 - 4 && kHaloWideTabMax < 2048 - 4, "groups and their padding fit the hash");
template <class V>
constexpr bool holds_overshoot = V::kTab + V::kCutAhead * V::kThreads < V::kHash;
static_assert(holds_overshoot<NarrowItem> && holds_overshoot<WideItem>, "add_rows' ids past the limit fit the hash");
static_assert(kHaloSlicesPerItem == kPick, "the cut's maps have 8 states");

static_assert(kHaloWideTabMax * 16 <= 0x3fff + 1, "a row's own offset fits the header's 14 bits");

// What the kernels report.
enum : uint32_t { kDoesNotFit = 1, kDisagree = 2 };
struct BuildTotals {
    unsigned long long words;
    unsigned long long ids;
    uint32_t items;
    uint32_t runs;
    uint32_t flags;
    uint32_t pad_;
};

// One item as cut_runs_kernel finds it, at its first block.
struct CutItem {
    uint32_t blocks;
    uint32_t ntab;
    uint32_t words;
};

// ---- the cut into runs
// A run ends at most 8 blocks after its start, so a tile of blocks is a map
// from the block at which a run enters it (0 .. 7 after its first) to the one
// at which the next tile is entered: 3 bits for each of 8 entries.
constexpr int kRunTile = 256;

__device__ __forceinline__ uint32_t compose(uint32_t first, uint32_t then)
{
    uint32_t r = 0;
#pragma unroll
    for (int e = 0; e < kPick; e++) r |= ((then >> (3 * ((first >> (3 * e)) & 7u))) & 7u) << (3 * e);
    return r;
}

// run[q] = blocks of the run that starts at block q (at most 8, at most
// `stream` words), and each tile's map.
__global__ void __launch_bounds__(kRunTile) block_runs_kernel(const uint32_t* __restrict__ row_off, int64_t n,
                                                             int64_t blocks, uint32_t stream,
                                                             uint8_t* __restrict__ run, uint32_t* __restrict__ map,
                                                             BuildTotals* out)
{
    __shared__ uint32_t words[kRunTile + kPick];
    __shared__ uint8_t len_s[kRunTile];
    __shared__ uint32_t exits;
    const int64_t tiles = (blocks + kRunTile - 1) / kRunTile;
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int64_t q0 = t * kRunTile;
        for (int k = threadIdx.x; k < kRunTile + kPick; k += kRunTile) {
            const int64_t q = q0 + k;
            uint32_t w = 0xffffffffu;  // past the end: never taken
            if (q < blocks) {
                uint32_t longest = 0, a = row_off[8 * q];
                for (int64_t r = 8 * q + 1; r <= min(8 * q + 8, n); r++) {
                    const uint32_t b = row_off[r];
                    longest = max(longest, b - a);
                    a = b;
                }
                const uint64_t wq = 32ull * (((uint64_t)longest + 7) / 8 + 1);
                if (wq > stream || longest > 1023u) atomicOr(&out->flags, kDoesNotFit);  // 10 bits of the header
                w = (uint32_t)min(wq, (uint64_t)0xfffffff0u);
            }
            words[k] = w;
        }
        if (threadIdx.x == 0) exits = 0;
        __syncthreads();
        const int size = (int)min((int64_t)kRunTile, blocks - q0);
        if ((int)threadIdx.x < size) {
            uint64_t sum = words[threadIdx.x];
            int len = 1;
            while (len < kPick && sum + words[threadIdx.x + len] <= stream) sum += words[threadIdx.x + len++];
            run[q0 + threadIdx.x] = (uint8_t)len;
            len_s[threadIdx.x] = (uint8_t)len;
        }
        __syncthreads();
        if (threadIdx.x < kPick) {
            int q = threadIdx.x;
            while (q < size) q += len_s[q];
            atomicOr(&exits, (uint32_t)((q - size) & 7) << (3 * threadIdx.x));
        }
        __syncthreads();
        if (threadIdx.x == 0) map[t] = exits;
        __syncthreads();
    }
}

// One CTA: enter[t] = the block of tile t at which a run starts first.
__global__ void __launch_bounds__(1024) run_entries_kernel(const uint32_t* __restrict__ map, int64_t tiles,
                                                          uint8_t* __restrict__ enter)
{
    __shared__ uint32_t part[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t identity = 076543210u;
    const int64_t chunk = (tiles + 1023) / 1024;
    const int64_t c0 = min(tid * chunk, tiles), c1 = min(c0 + chunk, tiles);
    uint32_t inc = identity;
    for (int64_t t = c0; t < c1; t++) inc = compose(inc, map[t]);
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc = compose(o, inc);
    }
    if (lane == 31) part[warp] = inc;
    __syncthreads();
    uint32_t before = identity;
    for (int w = 0; w < warp; w++) before = compose(before, part[w]);
    const uint32_t prev = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane) before = compose(before, prev);
    for (int64_t t = c0; t < c1; t++) {  // from block 0 of tile 0
        enter[t] = (uint8_t)(before & 7u);
        before = compose(before, map[t]);
    }
}

// One warp per tile: its runs' first blocks into the list (in any order).
__global__ void __launch_bounds__(kRunTile) list_runs_kernel(const uint8_t* __restrict__ run,
                                                            const uint8_t* __restrict__ enter, int64_t blocks,
                                                            int32_t* __restrict__ list, BuildTotals* out)
{
    __shared__ uint8_t len_s[kRunTile / 32][kRunTile];
    __shared__ uint8_t at_s[kRunTile / 32][kRunTile];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t tiles = (blocks + kRunTile - 1) / kRunTile;
    for (int64_t t = (int64_t)blockIdx.x * (kRunTile / 32) + warp; t < tiles; t += (int64_t)gridDim.x * (kRunTile / 32)) {
        const int64_t q0 = t * kRunTile;
        const int size = (int)min((int64_t)kRunTile, blocks - q0);
        for (int k = lane; k < size; k += 32) len_s[warp][k] = run[q0 + k];
        __syncwarp();
        int count = 0;
        if (lane == 0)
            for (int q = enter[t]; q < size; q += len_s[warp][q]) at_s[warp][count++] = (uint8_t)q;
        count = __shfl_sync(0xffffffffu, count, 0);
        uint32_t to = 0;
        if (lane == 0) to = atomicAdd(&out->runs, (uint32_t)count);
        to = __shfl_sync(0xffffffffu, to, 0);
        __syncwarp();
        for (int k = lane; k < count; k += 32) list[to + k] = (int32_t)(q0 + at_s[warp][k]);
        __syncwarp();
    }
}

// ---- the table of a set of rows: a hash of 32-id groups
// Buckets of two keys, read together: with ~120 groups in 512 buckets nearly
// every group sits in its own bucket, so the lanes of a warp do not wait for
// one another's probes.
template <int HASH>
struct GroupSet {
    int2 key[HASH / 2];    // id / 32 of a bucket's two groups, -1: free
    uint2 group[HASH];     // x: the group's ids in the set, y: its first slot (once known)

    static __device__ __forceinline__ uint32_t bucket(int32_t group)
    {
        return ((uint32_t)group * 2654435761u) >> (HASH == 1024 ? 23 : 22);
    }
    // Adds id; true if it was new; at: the group's place.  At most HASH - 1
    // groups may ever be held.
    __device__ __forceinline__ bool add(int32_t id, uint32_t& at)
    {
        const int32_t group = id >> 5;
        const uint32_t bit = 1u << (id & 31);
        uint32_t h = bucket(group);
        for (int probes = 0;; probes++) {
            if (probes == HASH / 2) return false;  // full: not reached, see add_rows
            int2 k;
            asm volatile("ld.volatile.shared.v2.s32 {%0, %1}, [%2];"
                         : "=r"(k.x), "=r"(k.y)
                         : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(&key[h]))));
            at = 2 * h;
            if (k.x == group) break;
            at++;
            if (k.y == group) break;
            if (k.x == -1) {
                k.x = atomicCAS(&key[h].x, -1, group);
                at--;
                if (k.x == -1 || k.x == group) break;
                at++;
            }
            if (k.y == -1) {
                k.y = atomicCAS(&key[h].y, -1, group);
                if (k.y == -1 || k.y == group) break;
            }
            h = (h + 1) & (HASH / 2 - 1);
        }
        uint32_t* const mask = &this->group[at].x;
        if (*(volatile uint32_t*)mask & bit) return false;
        return !(atomicOr(mask, bit) & bit);
    }
    // The slot of an id of the group at `at`: the group's first slot plus the
    // ids before it.
    __device__ __forceinline__ uint32_t slot(uint32_t at, uint32_t id) const
    {
        const uint2 g = group[at];
        return g.y + (uint32_t)__popc(g.x & ((1u << (id & 31u)) - 1u));
    }
    __device__ __forceinline__ uint32_t find(int32_t group) const  // held
    {
        uint32_t h = bucket(group);
        for (int probes = 0; probes < HASH / 2; probes++) {
            const int2 k = key[h];
            if (k.x == group) return 2 * h;
            if (k.y == group) return 2 * h + 1;
            h = (h + 1) & (HASH / 2 - 1);
        }
        return 0;  // not held: not reached
    }
    __device__ __forceinline__ int32_t key_at(int k) const { return k & 1 ? key[k / 2].y : key[k / 2].x; }
    __device__ __forceinline__ void clear()
    {
        for (int k = threadIdx.x; k < HASH; k += blockDim.x) {
            if (!(k & 1)) key[k / 2] = make_int2(-1, -1);
            group[k] = make_uint2(0, 0);
        }
    }
};

// Adds the ids of rows [r0, r1) -- the rows and their columns -- and counts
// the new ones in *count, giving up once it is above `most`.  loc, if given,
// gets for each entry its group's place | (id mod 32) << 11.  Whole CTA; each
// thread has kAhead columns in flight, so up to kAhead ids per thread are added
// past `most`: the hash holds them.
template <int kAhead, int HASH>
__device__ __forceinline__ void add_rows(GroupSet<HASH>& set, const uint32_t* __restrict__ row_off,
                                         const int32_t* __restrict__ col, int64_t r0, int64_t r1, int* count,
                                         int most, uint16_t* loc)
{
    const uint32_t e0 = row_off[r0], m = row_off[r1] - e0;
    const uint32_t rows = (uint32_t)(r1 - r0), step = blockDim.x;
    const int lane = threadIdx.x & 31;
    uint32_t at;
    for (uint32_t k0 = threadIdx.x & ~31u; k0 < rows; k0 += step) {
        const bool fresh = k0 + lane < rows && set.add((int32_t)(r0 + k0 + lane), at);
        const uint32_t b = __ballot_sync(0xffffffffu, fresh);
        if (lane == 0 && b) atomicAdd(count, __popc(b));
    }
    for (uint32_t k0 = threadIdx.x & ~31u; k0 < m; k0 += kAhead * step) {
        if (__any_sync(0xffffffffu, *(volatile int*)count > most)) return;
        int32_t id[kAhead];
#pragma unroll
        for (int x = 0; x < kAhead; x++) {
            const uint32_t k = k0 + x * step + lane;
            id[x] = k < m ? col[e0 + k] : -1;
        }
        int news = 0;
#pragma unroll
        for (int x = 0; x < kAhead; x++) {
            if (id[x] >= 0) {
                news += set.add(id[x], at) ? 1 : 0;
                if (loc) loc[k0 + x * step + lane] = (uint16_t)(at | ((uint32_t)(id[x] & 31) << 11));
            }
        }
        news = __reduce_add_sync(0xffffffffu, news);
        if (lane == 0 && news) atomicAdd(count, news);
    }
}

// Row lengths of an item ordered longest first, ties by row: rank of row k of m.
__device__ __forceinline__ int length_rank(const uint32_t* len, int m, int k)
{
    const uint32_t mine = len[k];
    int rank = 0;
    for (int x = 0; x < m; x++) rank += (len[x] > mine || (len[x] == mine && x < k)) ? 1 : 0;
    return rank;
}

// One CTA per run: its items.  A run whose table fits is one item; else the
// longest prefixes that fit, block by block.
template <class V>
__global__ void __launch_bounds__(V::kThreads) cut_runs_kernel(const uint32_t* __restrict__ row_off,
                                                              const int32_t* __restrict__ col, int64_t n,
                                                              const int32_t* __restrict__ list,
                                                              const uint8_t* __restrict__ run,
                                                              CutItem* __restrict__ cut,
                                                              uint8_t* __restrict__ cuts, BuildTotals* out)
{
    __shared__ GroupSet<V::kHash> set;
    __shared__ uint32_t len[8 * kPick];
    __shared__ int count;
    __shared__ uint32_t words;
    if (out->flags) return;
    const uint32_t runs = out->runs;
    for (uint32_t r = blockIdx.x; r < runs; r += gridDim.x) {
        const int64_t b0 = list[r];
        const int nb = run[b0];
        const int64_t b1 = b0 + nb;
        int from = 0;
        while (from < nb) {
            // all that is left at once; if that does not fit, block by block
            int to = nb, ntab = 0;
            for (int whole = 1; whole >= 0; whole--) {
                __syncthreads();
                set.clear();
                if (threadIdx.x == 0) count = 0;
                __syncthreads();
                if (whole) {
                    add_rows<V::kCutAhead>(set, row_off, col, 8 * (b0 + from), min(8 * b1, n), &count, V::kTab, nullptr);
                    __syncthreads();
                    ntab = count;
                    if (ntab <= V::kTab) break;
                } else {
                    for (to = from; to < nb; to++) {
                        add_rows<V::kCutAhead>(set, row_off, col, 8 * (b0 + to), min(8 * (b0 + to + 1), n), &count, V::kTab, nullptr);
                        __syncthreads();
                        const int c = count;
                        __syncthreads();
                        if (c > V::kTab) break;
                        ntab = c;
                    }
                }
            }
            if (to == from) {  // one block's table is too large
                if (threadIdx.x == 0) atomicOr(&out->flags, kDoesNotFit);
                return;
            }
            // the item's words: slice j is as long as the row of rank 8 j
            const int64_t r0 = 8 * (b0 + from);
            const int m = (int)(min(8 * (b0 + to), n) - r0);
            __syncthreads();
            if ((int)threadIdx.x < m) len[threadIdx.x] = row_off[r0 + threadIdx.x + 1] - row_off[r0 + threadIdx.x];
            if (threadIdx.x == 0) words = 0;
            __syncthreads();
            if ((int)threadIdx.x < m && (length_rank(len, m, threadIdx.x) & 7) == 0)
                atomicAdd(&words, 32u * ((len[threadIdx.x] + 7u) / 8u + 1u));
            __syncthreads();
            if (threadIdx.x == 0)
                cut[b0 + from] = CutItem{(uint32_t)(to - from), (uint32_t)ntab, words};
            if (threadIdx.x == 0) cuts[b0 + from] = 1;
            from = to;
        }
    }
}

// The items in row order with their places in the words and tables: each CTA
// takes a stretch of the blocks, sums its items (WRITE false), then writes them
// after the sums of the stretches before it (true).
constexpr int kPlaceThreads = 256, kPlaceCtas = 64;
struct Places {
    unsigned long long items, ids, words;
};

template <bool WRITE>
__global__ void __launch_bounds__(kPlaceThreads) place_items_kernel(int64_t n, int64_t blocks,
                                                                   const CutItem* __restrict__ cut,
                                                                   const uint8_t* __restrict__ cuts,
                                                                   Places* __restrict__ sums,
                                                                   WorkItem* __restrict__ items, BuildTotals* out)
{
    constexpr int kWarps = kPlaceThreads / 32;
    __shared__ Places tot[kWarps + 1];
    if (out->flags) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t stretch = (blocks + gridDim.x - 1) / gridDim.x;
    const int64_t s0 = min(blockIdx.x * stretch, blocks), s1 = min(s0 + stretch, blocks);
    Places base{0, 0, 0};
    if (WRITE) {
        for (unsigned c = 0; c < blockIdx.x; c++) {
            base.items += sums[c].items;
            base.ids += sums[c].ids;
            base.words += sums[c].words;
        }
    }
    for (int64_t t0 = s0; t0 < s1; t0 += kPlaceThreads) {
        const int64_t q = t0 + tid;
        const bool is = q < s1 && cuts[q];
        CutItem c{0, 0, 0};
        if (is) c = cut[q];
        Places v{is ? 1ull : 0ull, c.ntab, c.words};
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned long long a = __shfl_up_sync(0xffffffffu, v.items, off);
            const unsigned long long b = __shfl_up_sync(0xffffffffu, v.ids, off);
            const unsigned long long d = __shfl_up_sync(0xffffffffu, v.words, off);
            if (lane >= off) {
                v.items += a;
                v.ids += b;
                v.words += d;
            }
        }
        __syncthreads();
        if (lane == 31) tot[warp] = v;
        __syncthreads();
        Places before = base;
        for (int x = 0; x < kWarps; x++) {
            const Places y = tot[x];
            if (x < warp) {
                before.items += y.items;
                before.ids += y.ids;
                before.words += y.words;
            }
            base.items += y.items;
            base.ids += y.ids;
            base.words += y.words;
        }
        if (WRITE && is) {
            WorkItem w{};
            w.row0 = (int32_t)(8 * q);
            w.nrows = (int32_t)(min(8 * (q + c.blocks), n) - 8 * q);
            w.flags = kItemStaged;
            w.nent = c.words;
            w.ent0 = (uint32_t)(before.words + v.words - c.words);
            w.ntab = c.ntab;
            w.tab0 = (uint32_t)(before.ids + v.ids - c.ntab);
            items[before.items + v.items - 1] = w;
        }
    }
    if (tid == 0) {
        if (!WRITE) {
            sums[blockIdx.x] = base;
        } else if (blockIdx.x == gridDim.x - 1) {
            out->items = (uint32_t)base.items;
            out->ids = base.ids;
            out->words = base.words;
        }
    }
}

// One CTA per item: its sorted table into ids[tab0, tab0 + ntab), its slices'
// offsets, and the words of its slices.
template <class V>
__global__ void __launch_bounds__(V::kThreads, V::kCtas) fill_items_kernel(
    const uint32_t* __restrict__ row_off, const int32_t* __restrict__ col, int num_items,
    const WorkItem* __restrict__ items, uint32_t* __restrict__ slice_off, int32_t* __restrict__ ids,
    uint32_t* __restrict__ words, BuildTotals* out)
{
    constexpr int kWarps = V::kThreads / 32;
    constexpr int kEntries = 2 * V::kStream;  // every word of a step holds two entries
    extern __shared__ __align__(16) unsigned char dyn[];
    // [kEntries] per row: its entries' groups (add_rows), then, in place, their
    // slots bucketed by bank group
    uint16_t* const rs = reinterpret_cast<uint16_t*>(dyn);
    __shared__ GroupSet<V::kHash> set;
    __shared__ __align__(16) int32_t gid[V::kHash];  // the groups, as collected
    __shared__ uint16_t gat[V::kHash];          // their places
    __shared__ uint16_t sorted[V::kHash];       // collected index of the k-th group
    __shared__ uint32_t off[8 * kPick + 1];     // the rows' first entries, from the item's
    __shared__ uint32_t len[8 * kPick];
    __shared__ int order[8 * kPick];            // the item's rows, longest first
    __shared__ uint32_t at[kPick + 1];          // the slices' first words, from the item's
    __shared__ uint16_t bucket[8 * kPick][8];   // a row's buckets: first places in rs
    __shared__ uint32_t part[kWarps];
    __shared__ int count;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int item = blockIdx.x; item < num_items; item += gridDim.x) {
        const WorkItem w = items[item];
        const int m = w.nrows, ns = (m + 7) / 8;
        __syncthreads();
        set.clear();
        if (tid == 0) count = 0;
        const uint32_t e0 = row_off[w.row0];
        if (tid <= m) off[tid] = row_off[w.row0 + tid] - e0;
        __syncthreads();
        if (tid < m) len[tid] = off[tid + 1] - off[tid];
        const bool fits = off[m] <= (uint32_t)kEntries;
        if (fits) add_rows<4>(set, row_off, col, w.row0, (int64_t)w.row0 + m, &count, V::kTab, rs);
        __syncthreads();
        if (count != (int)w.ntab || !fits) {  // the cut and the fill disagree
            if (tid == 0) atomicOr(&out->flags, kDisagree);
            continue;
        }
        __syncthreads();
        if (tid == 0) count = 0;
        __syncthreads();
        // the groups, then in order (each counts the smaller ones), and each
        // one's first slot
        for (int k = tid; k < V::kHash; k += V::kThreads) {
            const int32_t g = set.key_at(k);
            if (g != -1) {
                const int x = atomicAdd(&count, 1);
                gid[x] = g;
                gat[x] = (uint16_t)k;
            }
        }
        if (tid < m) order[length_rank(len, m, tid)] = tid;
        __syncthreads();
        const int groups = count;
        if (tid < 4) gid[groups + tid] = INT_MAX;  // whole reads of four (groups < kHash - 4: kTab is)
        if (warp == kWarps - 1 && lane < 8) {
            const uint32_t words_j = lane < ns ? 32u * ((len[order[8 * lane]] + 7u) / 8u + 1u) : 0u;
            uint32_t sum = words_j;
            for (int x = 1; x < 8; x <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffu, sum, x);
                if (lane >= x) sum += y;
            }
            if (lane == 0) at[0] = 0;
            if (lane < ns) at[lane + 1] = sum;
        }
        __syncthreads();
        for (int k = tid; k < groups; k += V::kThreads) {
            const int32_t g = gid[k];
            int rank = 0;
            for (int x = 0; x < groups; x += 4) {
                const int4 y = *reinterpret_cast<const int4*>(gid + x);
                rank += (y.x < g) + (y.y < g) + (y.z < g) + (y.w < g);
            }
            sorted[rank] = (uint16_t)k;
        }
        __syncthreads();
        uint32_t base = 0;
        for (int k0 = 0; k0 < groups; k0 += V::kThreads) {
            const int k = k0 + tid;
            const int x0 = k < groups ? sorted[k] : 0;
            const uint32_t place = gat[x0];
            const uint32_t mask = k < groups ? set.group[place].x : 0u;
            const uint32_t mine = __popc(mask);
            uint32_t sum = mine;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += y;
            }
            if (lane == 31) part[warp] = sum;
            __syncthreads();
            uint32_t slot = base + sum - mine;
            for (int x = 0; x < warp; x++) slot += part[x];
            for (int x = 0; x < kWarps; x++) base += part[x];
            if (k < groups) {
                set.group[place].y = slot;
                const int32_t id0 = gid[x0] << 5;
                for (uint32_t b = mask; b; b &= b - 1) ids[(int64_t)w.tab0 + slot++] = id0 + __ffs(b) - 1;
            }
            __syncthreads();
        }
        auto slot_of = [&](int32_t id) { return set.slot(set.find(id >> 5), (uint32_t)id); };
        // one warp per row: its entries' slots bucketed by bank group, each
        // bucket ascending (the row's columns are).  Lane g (mod 8) counts
        // group g.  A row of up to kHeld * 32 entries stays in registers, each
        // entry with its rank in its bucket, between counting and placing; a
        // longer one reads its columns again.
        for (int r = warp; r < m; r += kWarps) {
            const uint32_t o = off[r], l = len[r];
            uint32_t total = 0;
            // rank of the lane's slot in its bucket; counts the buckets on
            auto rank_of = [&](uint32_t sl, bool v) {
                const uint32_t bv = __ballot_sync(0xffffffffu, v), b0 = __ballot_sync(0xffffffffu, sl & 1u),
                               b1 = __ballot_sync(0xffffffffu, sl & 2u), b2 = __ballot_sync(0xffffffffu, sl & 4u);
                const uint32_t peers = bv & (sl & 1u ? b0 : ~b0) & (sl & 2u ? b1 : ~b1) & (sl & 4u ? b2 : ~b2);
                const uint32_t mine = bv & (lane & 1 ? b0 : ~b0) & (lane & 2 ? b1 : ~b1) & (lane & 4 ? b2 : ~b2);
                const uint32_t before = __shfl_sync(0xffffffffu, total, sl & 7u);
                total += __popc(mine);
                return before + __popc(peers & ((1u << lane) - 1u));
            };
            auto starts_of = [&]() {  // of group (lane mod 8)
                uint32_t sum = total;
                for (int x = 1; x < 8; x <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, sum, x, 8);
                    if ((lane & 7) >= x) sum += y;
                }
                const uint32_t start = o + sum - total;
                if (lane < 8) bucket[r][lane] = (uint16_t)start;
                return start;
            };
            if (l <= 32u * V::kHeld) {
                uint32_t held[V::kHeld];  // slot | rank << 16
#pragma unroll
                for (int x = 0; x < V::kHeld; x++)
                    if (32u * x < l) {
                        const bool v = 32u * x + lane < l;
                        const uint32_t e = v ? rs[o + 32 * x + lane] : 0u;
                        const uint32_t sl = set.slot(e & 2047u, e >> 11);
                        held[x] = sl | (rank_of(sl, v) << 16);
                    }
                const uint32_t start = starts_of();
                __syncwarp();
#pragma unroll
                for (int x = 0; x < V::kHeld; x++)
                    if (32u * x < l) {
                        const uint32_t to = __shfl_sync(0xffffffffu, start, held[x] & 7u);
                        if (32u * x + lane < l) rs[to + (held[x] >> 16)] = (uint16_t)held[x];
                    }
            } else {
                const int32_t* __restrict__ row = col + e0 + o;
                for (uint32_t k0 = 0; k0 < l; k0 += 32) {
                    const bool v = k0 + lane < l;
                    rank_of(v ? slot_of(row[k0 + lane]) : 0u, v);
                }
                const uint32_t start = starts_of();
                total = 0;
                __syncwarp();
                for (uint32_t k0 = 0; k0 < l; k0 += 32) {
                    const bool v = k0 + lane < l;
                    const uint32_t sl = v ? slot_of(row[k0 + lane]) : 0u;
                    const uint32_t rank = rank_of(sl, v);
                    const uint32_t to = __shfl_sync(0xffffffffu, start, sl & 7u);
                    if (v) rs[to + rank] = (uint16_t)sl;
                }
            }
        }
        __syncthreads();
        if (tid < ns) slice_off[w.row0 / 8 + tid + 1] = w.ent0 + at[tid + 1];
        if (tid == 0 && w.row0 == 0) slice_off[0] = 0;
        // one thread per row position: the picks
        if (tid < 8 * ns) {
            const int j = tid / 8, i = tid & 7;
            const int T = (int)((at[j + 1] - at[j]) / 32) - 1;
            uint32_t* sw = words + w.ent0 + at[j];
            uint32_t own = 0;
            uint32_t hdr = 1u << 31;  // a padding row
            // st[c]: a bank group's state, left << 19 | (7 - group) << 16 | next
            // place in the row's part of rs: the largest of them is the fullest
            // group, the first such on ties.  Position c is group (c + 2t + 4p)
            // mod 8 in step t: a step shifts the window by two groups, so the
            // states are shifted instead and every index is a constant.
            constexpr uint32_t kOne = 1u << 19;
            const uint32_t p4 = 4u * (i & 1);
            uint32_t st[8];
            uint32_t o = 0;
#pragma unroll
            for (int c = 0; c < 8; c++) st[c] = 0;
            if (tid < m) {
                const int lrow = order[tid];
                const uint32_t l = len[lrow];
                o = off[lrow];
                own = slot_of(w.row0 + lrow) * 16u;
                hdr = own | (l << 14) | ((uint32_t)lrow << 24);
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const uint32_t g = (c + p4) & 7u;
                    const uint32_t a = bucket[lrow][g], b = g == 7u ? o + l : bucket[lrow][g + 1];
                    st[c] = ((b - a) << 19) | ((7u - g) << 16) | (a - o);
                }
            }
            const uint16_t* row = rs + o;
            *reinterpret_cast<uint4*>(sw + 4 * i) = make_uint4(hdr, hdr, hdr, hdr);
            for (int t = 0; t < T; t++) {
                uint32_t pk[2][4];
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int l = 0; l < 4; l++) {
                        // the window's group if its bucket has slots left, else
                        // the fullest, else padding (the row's own slot)
                        uint32_t take = st[h + l];
                        if (take < kOne)
                            take = max(max(max(st[0], st[1]), max(st[2], st[3])),
                                       max(max(st[4], st[5]), max(st[6], st[7])));
                        pk[h][l] = own;
                        if (take >= kOne) {
                            pk[h][l] = 16u * row[take & 0xffffu];
#pragma unroll
                            for (int x = 0; x < 8; x++)
                                if (st[x] == take) st[x] += 1u - kOne;
                        }
                    }
                *reinterpret_cast<uint4*>(sw + 32 * (t + 1) + 4 * i) =
                    make_uint4(pk[0][0] | (pk[1][0] << 16), pk[0][1] | (pk[1][1] << 16),
                               pk[0][2] | (pk[1][2] << 16), pk[0][3] | (pk[1][3] << 16));
                const uint32_t s0 = st[0], s1 = st[1];
#pragma unroll
                for (int x = 0; x < 6; x++) st[x] = st[x + 2];
                st[6] = s0;
                st[7] = s1;
            }
        }
    }
}

template <class T>
cudaError_t alloc_n(T** p, int64_t count, cudaStream_t s)
{
    return irr_malloc_async(p, sizeof(T) * (size_t)(count > 0 ? count : 1), s);
}

template <class V>
cudaError_t build(const uint32_t* row_off, const int32_t* col, int64_t n, Staged* st, cudaStream_t s)
{
    const int64_t S = (n + 7) / 8;
    int dev = 0, sms = 0;
    IRR_CUDA_TRY(cudaGetDevice(&dev));
    IRR_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int64_t tiles = (S + kRunTile - 1) / kRunTile;
    uint8_t *run = nullptr, *cuts = nullptr, *enter = nullptr;
    uint32_t* map = nullptr;
    int32_t* list = nullptr;
    CutItem* cut = nullptr;
    Places* sums = nullptr;
    WorkItem* items = nullptr;
    BuildTotals* d_out = nullptr;
    BuildTotals got{};
    Staged out;
    out.slices = S;
    out.wide = V::kTab > kHaloTabMax;
    auto go = [&]() -> cudaError_t {
        // runs and items are at most the blocks
        IRR_CUDA_TRY(alloc_n(&run, S, s));
        IRR_CUDA_TRY(alloc_n(&cuts, S, s));
        IRR_CUDA_TRY(alloc_n(&enter, tiles, s));
        IRR_CUDA_TRY(alloc_n(&map, tiles, s));
        IRR_CUDA_TRY(alloc_n(&list, S, s));
        IRR_CUDA_TRY(alloc_n(&cut, S, s));
        IRR_CUDA_TRY(alloc_n(&sums, kPlaceCtas, s));
        IRR_CUDA_TRY(alloc_n(&items, S, s));
        IRR_CUDA_TRY(alloc_n(&d_out, 1, s));
        IRR_CUDA_TRY(cudaMemsetAsync(d_out, 0, sizeof(BuildTotals), s));
        IRR_CUDA_TRY(cudaMemsetAsync(cuts, 0, (size_t)(S > 0 ? S : 1), s));
        if (S > 0) {
            block_runs_kernel<<<(unsigned)std::min<int64_t>(tiles, 8192), kRunTile, 0, s>>>(
                row_off, n, S, (uint32_t)V::kStream, run, map, d_out);
            run_entries_kernel<<<1, 1024, 0, s>>>(map, tiles, enter);
            list_runs_kernel<<<(unsigned)std::min<int64_t>((tiles + 7) / 8, 8192), kRunTile, 0, s>>>(run, enter, S,
                                                                                                    list, d_out);
            cut_runs_kernel<V><<<(unsigned)std::min<int64_t>(S, (int64_t)sms * 128), V::kThreads, 0, s>>>(
                row_off, col, n, list, run, cut, cuts, d_out);
            place_items_kernel<false><<<kPlaceCtas, kPlaceThreads, 0, s>>>(n, S, cut, cuts, sums, items, d_out);
            place_items_kernel<true><<<kPlaceCtas, kPlaceThreads, 0, s>>>(n, S, cut, cuts, sums, items, d_out);
            IRR_CUDA_TRY(cudaGetLastError());
        }
        IRR_CUDA_TRY(cudaMemcpyAsync(&got, d_out, sizeof(got), cudaMemcpyDeviceToHost, s));
        IRR_CUDA_TRY(cudaStreamSynchronize(s));
        if ((got.flags & kDoesNotFit) || got.words > 0xffffffffull || got.ids > 0x7fffffffull)
            return cudaErrorNotSupported;
        out.nwords = (int64_t)got.words;
        out.nids = (int64_t)got.ids;
        out.nitems = got.items;
        IRR_CUDA_TRY(alloc_n(&out.slice_off, S + 1, s));
        IRR_CUDA_TRY(alloc_n(&out.words, out.nwords, s));
        IRR_CUDA_TRY(alloc_n(&out.ids, out.nids, s));
        IRR_CUDA_TRY(alloc_n(&out.items, out.nitems, s));
        if (S == 0) IRR_CUDA_TRY(cudaMemsetAsync(out.slice_off, 0, sizeof(uint32_t), s));
        if (got.items > 0) {
            const int smem = 2 * V::kStream * (int)sizeof(uint16_t);
            IRR_CUDA_TRY(cudaMemcpyAsync(out.items, items, sizeof(WorkItem) * got.items, cudaMemcpyDeviceToDevice, s));
            IRR_CUDA_TRY(cudaFuncSetAttribute(fill_items_kernel<V>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            fill_items_kernel<V><<<(unsigned)std::min<int64_t>(got.items, (int64_t)sms * 128), V::kThreads, smem, s>>>(
                row_off, col, (int)got.items, out.items, out.slice_off, out.ids, out.words, d_out);
            IRR_CUDA_TRY(cudaGetLastError());
            IRR_CUDA_TRY(cudaMemcpyAsync(&got, d_out, sizeof(got), cudaMemcpyDeviceToHost, s));
            IRR_CUDA_TRY(cudaStreamSynchronize(s));
            if (got.flags) return cudaErrorInvalidValue;
        }
        return cudaSuccess;
    };
    const cudaError_t e = go();
    void* tmp[] = {run, cuts, enter, map, list, cut, sums, items, d_out};
    for (void* p : tmp)
        if (p) cudaFreeAsync(p, s);
    if (e != cudaSuccess) {
        free_staged(&out, s);
        return e;
    }
    *st = out;
    return cudaSuccess;
}

}  // namespace

void free_staged(Staged* st, cudaStream_t s)
{
    void* ps[4] = {st->slice_off, st->words, st->ids, st->items};
    for (void* p : ps)
        if (p) {
            if (s) cudaFreeAsync(p, s);
            else cudaFree(p);
        }
    *st = Staged{};
}

cudaError_t build_staged(const uint32_t* row_off, const int32_t* col, int64_t n, bool wide, Staged* st,
                         cudaStream_t s)
{
    free_staged(st, s);
    return wide ? build<WideItem>(row_off, col, n, st, s) : build<NarrowItem>(row_off, col, n, st, s);
}

cudaError_t staged_items_to_host(const WorkItem* d_items, int64_t count, std::vector<WorkItem>* items, cudaStream_t s)
{
    items->resize((size_t)count);
    if (count > 0)
        IRR_CUDA_TRY(cudaMemcpyAsync(items->data(), d_items, sizeof(WorkItem) * (size_t)count, cudaMemcpyDeviceToHost, s));
    return cudaStreamSynchronize(s);
}

}  // namespace irr
