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
//   cut_runs_kernel    one CTA per run: its items, their tables and every
//                      entry's place in its item's table (scratch);
//   place_items_kernel the items' places in the words and tables;
//   fill_items_kernel  one CTA per item: its table, words and slice offsets.
// The rows come in any order (the partitioner's slots, unsorted): a table is
// gathered as a hash of 32-id groups with a bit per id -- neighbours on the
// curve share groups, so ~465 ids are ~120 groups to order, and an id's slot is
// its group's first slot plus a population count -- and a row's places are
// ordered as bits of a 1,024-bit map.
// What bounds it: instruction issue (a hash probe, a bit and a pick per entry).
// 1,000,003 nodes at 64 neighbours: sorting the rows, counting the tables and
// filling, a table gathered in both, 353 + 172 + 721 us; now 323 + 288, and the
// rows (4 bytes an entry) are made from the layout when they are asked for.
#include <algorithm>
#include <climits>
#include <vector>

#include "irr_internal.cuh"

namespace irr {
namespace {

constexpr int kPick = 8;                         // slices of an item, blocks of a run: at most
// The limits of the two variants.  kAhead: columns that a thread adds to a table
// between two looks at whether it is full (1, 2 or 4).
struct NarrowItem {
    static constexpr int kTab = kHaloTabMax, kStream = kHaloStreamMax;
    static constexpr int kHash = 1024, kCutThreads = 160, kAhead = 2;
    static constexpr int kFillWarps = 2, kFillCtas = 18;
};
struct WideItem {
    static constexpr int kTab = kHaloWideTabMax, kStream = kHaloWideStreamMax;
    static constexpr int kHash = 2048, kCutThreads = 256, kAhead = 4;
    static constexpr int kFillWarps = 4, kFillCtas = 8;
};
// add_rows' ids past the limit (8 rows' own ids, then what is in flight) fit the hash
template <class V>
constexpr bool holds_overshoot = V::kTab + 8 + V::kAhead * V::kCutThreads < V::kHash;
static_assert(holds_overshoot<NarrowItem> && holds_overshoot<WideItem>, "add_rows' ids past the limit fit the hash");
static_assert(kHaloTabMax <= 1024 && kHaloWideTabMax <= 1024, "a row's places fit its bit map");
static_assert(kHaloSlicesPerItem == kPick, "the cut's maps have 8 states");

static_assert(kHaloWideTabMax * 16 <= 0x3fff + 1, "a row's own offset fits the header's 14 bits");

// What the kernels report.
enum : uint32_t { kDoesNotFit = 1, kDoesNotPay = 2, kNoScratch = 4 };
struct BuildTotals {
    unsigned long long words;
    unsigned long long ids;
    unsigned long long cut_ids;  // of the tables cut so far
    uint32_t items;
    uint32_t runs;
    uint32_t flags;
    uint32_t entries;  // of the largest item
    uint32_t scratch;  // kNoScratch (no reason to stop the cut)
};

// One item as cut_runs_kernel finds it, at its first block.
struct CutItem {
    uint32_t blocks;
    uint32_t ntab;
    uint32_t words;
    uint32_t pad;
    unsigned long long tab0;  // its table's place in the scratch
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
    // Adds id; returns its group's place.  A new group is counted in *groups;
    // at most HASH - 1 may ever be held.
    __device__ __forceinline__ uint32_t add(int32_t id, int* groups)
    {
        const int32_t group = id >> 5;
        const uint32_t h = bucket(group);
        const int2 k = read(h);
        uint32_t at = 2 * h + (k.x != group);
        if (k.x != group && k.y != group) at = insert(group, h, groups);
        uint32_t* const mask = &this->group[at].x;
        const uint32_t bit = 1u << (id & 31);
        if (!(*(volatile uint32_t*)mask & bit)) atomicOr(mask, bit);
        return at;
    }
    __device__ __forceinline__ int2 read(uint32_t h)
    {
        int2 k;
        asm volatile("ld.volatile.shared.v2.s32 {%0, %1}, [%2];"
                     : "=r"(k.x), "=r"(k.y)
                     : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(&key[h]))));
        return k;
    }
    __device__ __forceinline__ uint32_t insert(int32_t group, uint32_t h, int* groups)
    {
        for (int probes = 0; probes < HASH / 2; probes++) {
            int2 k = read(h);
            if (k.x == -1) {
                k.x = atomicCAS(&key[h].x, -1, group);
                if (k.x == -1) {
                    atomicAdd(groups, 1);
                    return 2 * h;
                }
            }
            if (k.x == group) return 2 * h;
            if (k.y == -1) {
                k.y = atomicCAS(&key[h].y, -1, group);
                if (k.y == -1) {
                    atomicAdd(groups, 1);
                    return 2 * h + 1;
                }
            }
            if (k.y == group) return 2 * h + 1;
            h = (h + 1) & (HASH / 2 - 1);
        }
        return 0;  // full: not reached, see add_rows
    }
    // The slot of an id of the group at `at`: the group's first slot plus the
    // ids before it.
    __device__ __forceinline__ uint32_t slot(uint32_t at, uint32_t id) const
    {
        const uint2 g = group[at];
        return g.y + (uint32_t)__popc(g.x & ((1u << (id & 31u)) - 1u));
    }
    __device__ __forceinline__ int32_t key_at(int k) const { return k & 1 ? key[k / 2].y : key[k / 2].x; }
    __device__ __forceinline__ void clear()
    {
        for (int k = threadIdx.x; k < HASH / 4; k += blockDim.x)
            reinterpret_cast<int4*>(key)[k] = make_int4(-1, -1, -1, -1);
        for (int k = threadIdx.x; k < HASH / 2; k += blockDim.x)
            reinterpret_cast<uint4*>(group)[k] = make_uint4(0, 0, 0, 0);
    }
};

// An item's rows by two at a time, a half-warp each: f(entry, column) for each
// entry of rows [r0, r0 + rows), 4 columns of a thread read ahead, and after
// each kStep of them the whole warp calls go_on(), which may end it.
template <int kStep, class Each, class GoOn>
__device__ __forceinline__ void each_entry(const RowSource& src, int64_t r0, int rows, Each f, GoOn go_on)
{
    const int lane = threadIdx.x & 31, l = lane & 15;
    for (int p = (threadIdx.x >> 5) * 2; p < rows; p += (blockDim.x >> 5) * 2) {
        const int k = p + (lane >> 4);
        const int64_t r = r0 + k;
        uint32_t beg = 0, len = 0;
        if (k < rows) {
            beg = src.row_off[r];
            len = src.row_off[r + 1] - beg;
        }
        const int32_t* __restrict__ row = src.row(r, beg);
        const uint32_t longest = max(len, __shfl_xor_sync(0xffffffffu, len, 16));
        for (uint32_t x0 = l; x0 < longest + l; x0 += 64) {
            int32_t id[4];
#pragma unroll
            for (int x = 0; x < 4; x++) id[x] = x0 + 16 * x < len ? row[x0 + 16 * x] : -1;
#pragma unroll
            for (int x = 0; x < 4; x++) {
                if (id[x] >= 0) f(beg + x0 + 16 * x, id[x]);
                if (x % kStep == kStep - 1 && !go_on()) return;
            }
        }
    }
}

// place[e] = f(place[e]), each thread for the entries that each_entry gives it.
template <class F>
__device__ __forceinline__ void place_slots(const uint32_t* __restrict__ row_off, int64_t r0, int rows,
                                            uint16_t* place, F f)
{
    const int lane = threadIdx.x & 31, l = lane & 15;
    for (int p = (threadIdx.x >> 5) * 2; p < rows; p += (blockDim.x >> 5) * 2) {
        const int k = p + (lane >> 4);
        if (k >= rows) continue;
        const uint32_t beg = row_off[r0 + k], end = row_off[r0 + k + 1];
        uint32_t e = beg + l;
        for (; e + 48 < end; e += 64) {
            uint32_t u[4];
#pragma unroll
            for (int x = 0; x < 4; x++) u[x] = place[e + 16 * x];
#pragma unroll
            for (int x = 0; x < 4; x++) place[e + 16 * x] = f(u[x]);
        }
        for (; e < end; e += 16) place[e] = f(place[e]);
    }
}

// Adds the ids of rows [r0, r0 + rows) -- the rows and their columns --,
// giving up once their groups (*groups) are more than `most` ids can be in.
// own and place get for each row and entry its group's place | (id mod 32) << 11.
// Whole CTA.
template <int kAhead, int HASH>
__device__ __forceinline__ void add_rows(GroupSet<HASH>& set, const RowSource& src, int64_t r0, int rows, int* groups,
                                         int most, uint16_t* own, uint16_t* place)
{
    static_assert(HASH <= 2048, "a group's place fits 11 bits");
    auto add = [&](int32_t id) { return (uint16_t)(set.add(id, groups) | ((uint32_t)(id & 31) << 11)); };
    if ((int)threadIdx.x < rows) own[r0 + threadIdx.x] = add((int32_t)(r0 + threadIdx.x));  // at most 64 rows
    each_entry<kAhead>(
        src, r0, rows, [&](uint32_t e, int32_t id) { place[e] = add(id); },
        [&]() { return !__any_sync(0xffffffffu, *(volatile int*)groups > most); });
}

// Row lengths of an item ordered longest first, ties by row: rank of row k of
// m.  key[x] = len << 6 | 63 - x, 0 past m, in whole fours.
__device__ __forceinline__ uint32_t length_key(uint32_t len, int k) { return (len << 6) | (63u - (uint32_t)k); }
__device__ __forceinline__ int length_rank(const uint32_t* key, int m, int k)
{
    const uint32_t mine = key[k];
    int rank = 0;
    for (int x = 0; x < m; x += 4) {
        const uint4 y = *reinterpret_cast<const uint4*>(key + x);
        rank += (y.x > mine) + (y.y > mine) + (y.z > mine) + (y.w > mine);
    }
    return rank;
}

// One CTA per run: its items.  A run whose table fits is one item; else the
// longest prefixes that fit, block by block.  An item's table goes to the next
// free place of tab (room ids in all: without room for a table the items are
// counted on, and the layout is not to be written), place[e] (of the items'
// entries) and own[r] (of its rows) are their places in it.  most_ids: once the
// tables hold more ids between them, the layout is refused (~0: never).
template <class V>
__global__ void __launch_bounds__(V::kCutThreads) cut_runs_kernel(RowSource src, int64_t n,
                                                                 const int32_t* __restrict__ list,
                                                                 const uint8_t* __restrict__ run,
                                                                 CutItem* __restrict__ cut,
                                                                 uint8_t* __restrict__ cuts, uint16_t* own,
                                                                 uint16_t* place, int32_t* __restrict__ tab,
                                                                 unsigned long long room, unsigned long long most_ids,
                                                                 BuildTotals* out)
{
    __shared__ __align__(16) GroupSet<V::kHash> set;
    __shared__ __align__(16) uint32_t gkey[V::kTab + 4];  // the groups: id / 32 << 6 | ids in the set
    __shared__ uint16_t gat[V::kTab];                     // their places in the hash
    __shared__ __align__(16) uint32_t key[8 * kPick];
    __shared__ int held, ngroups;  // groups in the hash, and collected
    __shared__ int count;          // ids
    __shared__ uint32_t words;
    __shared__ uint32_t refused;
    __shared__ unsigned long long tab0;
    const int tid = threadIdx.x;
    // other CTAs may raise the flag now: one thread looks, for all to leave or none
    if (tid == 0) refused = *(volatile uint32_t*)&out->flags;
    __syncthreads();
    if (refused) return;
    const uint32_t runs = out->runs;
    auto reset = [&]() {
        __syncthreads();
        set.clear();
        if (tid == 0) {
            held = 0;
            ngroups = 0;
            count = 0;
            words = 0;
        }
        __syncthreads();
    };
    // blocks [b0, b1) added: the ids in the set now, kTab + 1 if more than kTab
    auto add = [&](int64_t b0, int64_t b1) {
        const int64_t r0 = 8 * b0;
        add_rows<V::kAhead>(set, src, r0, (int)(min(8 * b1, n) - r0), &held, V::kTab, own, place);
        __syncthreads();
        if (held > V::kTab) return V::kTab + 1;
        int ids = 0;
        for (int k = tid; k < V::kHash; k += V::kCutThreads) ids += __popc(set.group[k].x);
        ids = __reduce_add_sync(0xffffffffu, ids);
        if ((tid & 31) == 0) atomicAdd(&count, ids);
        __syncthreads();
        return min(count, V::kTab + 1);
    };
    for (uint32_t r = blockIdx.x; r < runs; r += gridDim.x) {
        const int64_t b0 = list[r];
        const int nb = run[b0];
        int from = 0;
        while (from < nb) {
            if (from > 0) {  // (a run of one item does without)
                __syncthreads();
                if (tid == 0) refused = *(volatile uint32_t*)&out->flags;
                __syncthreads();
                if (refused) return;
            }
            // all that is left at once; if that does not fit, block by block
            int to = nb;
            reset();
            int ntab = add(b0 + from, b0 + nb);
            if (ntab > V::kTab) {
                reset();
                for (to = from; to < nb; to++) {
                    if (add(b0 + to, b0 + to + 1) > V::kTab) break;
                    __syncthreads();
                    if (tid == 0) count = 0;  // counted whole after each block
                }
                if (to == from) {  // one block's table is too large
                    if (tid == 0) atomicOr(&out->flags, kDoesNotFit);
                    return;
                }
                reset();
                ntab = add(b0 + from, b0 + to);
            }
            const int64_t r0 = 8 * (b0 + from);
            const int m = (int)(min(8 * (b0 + to), n) - r0);
            // the groups, and each one's first slot: the ids of those before it
            for (int k = tid; k < V::kHash; k += V::kCutThreads) {
                const int32_t g = set.key_at(k);
                if (g != -1) {
                    const int x = atomicAdd(&ngroups, 1);
                    gkey[x] = ((uint32_t)g << 6) | (uint32_t)__popc(set.group[k].x);
                    gat[x] = (uint16_t)k;
                }
            }
            if (tid == 0) tab0 = atomicAdd(&out->cut_ids, (unsigned long long)ntab);
            if (tid < 8 * kPick) key[tid] = tid < m ? length_key(src.row_off[r0 + tid + 1] - src.row_off[r0 + tid], tid) : 0u;
            __syncthreads();
            const int groups = ngroups;
            if (tid < 4) gkey[groups + tid] = 0xffffffffu;  // whole reads of four
            // the item's words: slice j is as long as the row of rank 8 j
            if (tid < m && (length_rank(key, m, tid) & 7) == 0) atomicAdd(&words, 32u * (((key[tid] >> 6) + 7u) / 8u + 1u));
            __syncthreads();
            const unsigned long long t0 = tab0;
            const bool fits = t0 + ntab <= room;
            for (int k = tid; k < groups; k += V::kCutThreads) {
                const uint32_t mine = gkey[k];
                uint32_t slot = 0;
                for (int x = 0; x < groups; x += 4) {
                    const uint4 y = *reinterpret_cast<const uint4*>(gkey + x);
                    slot += (y.x < mine ? y.x & 63u : 0u) + (y.y < mine ? y.y & 63u : 0u) +
                            (y.z < mine ? y.z & 63u : 0u) + (y.w < mine ? y.w & 63u : 0u);
                }
                const uint32_t at = gat[k];
                set.group[at].y = slot;
                const int32_t id0 = (int32_t)(mine >> 6) << 5;
                for (uint32_t b = fits ? set.group[at].x : 0u; b; b &= b - 1) tab[t0 + slot++] = id0 + __ffs(b) - 1;
            }
            __syncthreads();
            // places: each thread those that it wrote
            auto slot_of = [&](uint32_t u) { return (uint16_t)set.slot(u & 2047u, u >> 11); };
            if (tid < m) own[r0 + tid] = slot_of(own[r0 + tid]);
            place_slots(src.row_off, r0, m, place, slot_of);
            if (tid == 0) {
                cut[b0 + from] = CutItem{(uint32_t)(to - from), (uint32_t)ntab, words, 0u, t0};
                cuts[b0 + from] = 1;
                atomicMax(&out->entries, src.row_off[r0 + m] - src.row_off[r0]);
                if (t0 + ntab > most_ids) atomicOr(&out->flags, kDoesNotPay);
                if (!fits) atomicOr(&out->scratch, kNoScratch);
            }
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
        CutItem c{0, 0, 0, 0, 0};
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

// One warp: the row's places row[0, l) ordered by bank group (place mod 8),
// each group ascending, and each group's first index into first[8].  A place is
// a bit of a map, 32 words of up to 32 bits: 4 words per group, of 2^shift
// places each.  bits: the warp's map, all zero before and after.  Rows that
// name a node twice are sorted by a bitonic network (of exchanges in one
// direction, so that any length can be padded with what is never moved).
__device__ __forceinline__ void order_by_bank(uint16_t* row, uint32_t l, int shift, uint32_t* bits, uint16_t* first,
                                              int lane)
{
    bool twice = false;
    for (uint32_t k = lane; k < l; k += 32) {
        const uint32_t sl = row[k], q = sl >> 3;
        const uint32_t bit = 1u << (q & ((1u << shift) - 1u));
        twice |= (atomicOr(bits + (((sl & 7u) << 2) | (q >> shift)), bit) & bit) != 0;
    }
    twice = __any_sync(0xffffffffu, twice);
    __syncwarp();
    const uint32_t mine = bits[lane];
    bits[lane] = 0;
    if (!twice) {
        uint32_t sum = __popc(mine);
#pragma unroll
        for (int x = 1; x < 32; x <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, sum, x);
            if (lane >= x) sum += y;
        }
        uint16_t* to = row + (sum - __popc(mine));
        if (!(lane & 3)) first[lane >> 2] = (uint16_t)(sum - __popc(mine));
        const uint32_t base = ((uint32_t)(lane & 3) << (shift + 3)) | ((uint32_t)lane >> 2);
        for (uint32_t b = mine; b; b &= b - 1) *to++ = (uint16_t)(base + 8u * (uint32_t)(__ffs(b) - 1));
        __syncwarp();
        return;
    }
    auto order = [](uint32_t sl) { return ((sl & 7u) << 13) | (sl >> 3); };
    auto exchange = [&](uint32_t a, uint32_t b) {  // a < b
        const uint32_t x = row[a], y = row[b];
        if (order(x) > order(y)) {
            row[a] = (uint16_t)y;
            row[b] = (uint16_t)x;
        }
    };
    for (uint32_t size = 2; size < 2 * l; size <<= 1) {
        for (uint32_t k = lane; k < l; k += 32) {
            const uint32_t o = k ^ (size - 1);
            if (o > k && o < l) exchange(k, o);
        }
        __syncwarp();
        for (uint32_t stride = size >> 2; stride > 0; stride >>= 1) {
            for (uint32_t k = lane; k < l; k += 32) {
                const uint32_t o = k ^ stride;
                if (o > k && o < l) exchange(k, o);
            }
            __syncwarp();
        }
    }
    if (lane < 8) {
        uint32_t lo = 0, hi = l;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) / 2;
            if ((row[mid] & 7u) < (uint32_t)lane) lo = mid + 1;
            else hi = mid;
        }
        first[lane] = (uint16_t)lo;
    }
    __syncwarp();
}

// One CTA per item: its table into ids[tab0, tab0 + ntab), its slices' offsets,
// and the words of its slices.  A warp orders the places of its rows, then
// picks for them, a thread per row, without waiting for the other warps; the
// longest rows go to the first.
template <class V>
__global__ void __launch_bounds__(V::kFillWarps * 32, V::kFillCtas) fill_items_kernel(
    const uint32_t* __restrict__ row_off, const uint16_t* __restrict__ own_place, const uint16_t* __restrict__ place,
    const int32_t* __restrict__ tab, const CutItem* __restrict__ cut, int num_items,
    const WorkItem* __restrict__ items, uint32_t* __restrict__ slice_off, int32_t* __restrict__ ids, uint32_t* __restrict__ words)
{
    constexpr int kWarps = V::kFillWarps, kThreads = 32 * kWarps, kRows = 8 * kPick / kWarps;
    static_assert(kRows <= 32, "a thread per row of the warp");
    extern __shared__ __align__(16) unsigned char dyn[];
    // the entries' places, 16-byte aligned as in memory (of the largest item:
    // every word of a step holds two, so at most 2 kStream), then ordered in place
    uint16_t* const rs = reinterpret_cast<uint16_t*>(dyn);
    __shared__ uint32_t off[8 * kPick + 1];     // the rows' first entries in rs
    __shared__ __align__(16) uint32_t key[8 * kPick];
    __shared__ int order[8 * kPick];            // the item's rows, longest first
    __shared__ uint32_t at[kPick + 1];          // the slices' first words, from the item's
    __shared__ uint16_t bucket[8 * kPick][8];   // a row's bank groups: first places in its part of rs
    __shared__ uint32_t bits[kWarps][32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    bits[warp][lane] = 0;
    for (int item = blockIdx.x; item < num_items; item += gridDim.x) {
        const WorkItem w = items[item];
        const int m = w.nrows, ns = (m + 7) / 8;
        const int64_t e0 = row_off[w.row0], base = e0 & ~7ll;
        __syncthreads();
        {
            const int chunks = (int)((row_off[w.row0 + m] - base + 7) / 8);
            const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(rs));
            for (int k = tid; k < chunks; k += kThreads)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16u * k), "l"(place + base + 8 * k)
                             : "memory");
        }
        for (int k = tid; k <= m; k += kThreads) off[k] = (uint32_t)(row_off[w.row0 + k] - base);
        for (int k = tid; k < 8 * kPick; k += kThreads)
            key[k] = k < m ? length_key(row_off[w.row0 + k + 1] - row_off[w.row0 + k], k) : 0u;
        const int32_t* from = tab + cut[w.row0 / 8].tab0;
        for (uint32_t k = tid; k < w.ntab; k += kThreads) ids[(int64_t)w.tab0 + k] = from[k];
        __syncthreads();
        for (int k = tid; k < m; k += kThreads) order[length_rank(key, m, k)] = k;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (lane < 8) {  // each warp for itself: the same values
            uint32_t sum = lane < ns ? 32u * (((key[order[8 * lane]] >> 6) + 7u) / 8u + 1u) : 0u;
            for (int x = 1; x < 8; x <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffu, sum, x);
                if (lane >= x) sum += y;
            }
            if (lane == 0) at[0] = 0;
            if (lane < ns) at[lane + 1] = sum;
        }
        const int shift = w.ntab <= 256 ? 3 : (w.ntab <= 512 ? 4 : 5);
        for (int p = kRows * warp; p < min(m, kRows * (warp + 1)); p++) {
            const int r = order[p];
            order_by_bank(rs + off[r], off[r + 1] - off[r], shift, bits[warp], bucket[r], lane);
        }
        __syncwarp();
        for (int k = tid; k < ns; k += kThreads) slice_off[w.row0 / 8 + k + 1] = w.ent0 + at[k + 1];
        if (tid == 0 && w.row0 == 0) slice_off[0] = 0;
        // one thread per row position: the picks
        const int pos = kRows * warp + lane;
        if (lane < kRows && pos < 8 * ns) {
            const int j = pos / 8, i = pos & 7;
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
            if (pos < m) {
                const int lrow = order[pos];
                const uint32_t l = key[lrow] >> 6;
                o = off[lrow];
                own = own_place[w.row0 + lrow] * 16u;
                hdr = own | (l << 14) | ((uint32_t)lrow << 24);
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const uint32_t g = (c + p4) & 7u;
                    const uint32_t a = bucket[lrow][g], b = g == 7u ? l : bucket[lrow][g + 1];
                    st[c] = ((b - a) << 19) | ((7u - g) << 16) | a;
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
cudaError_t build(const RowSource& src, int64_t n, int64_t m, int64_t most_ids, int64_t room, Staged* st, cudaStream_t s)
{
    const uint32_t* row_off = src.row_off;
    const int64_t S = (n + 7) / 8;
    // the narrow cut goes on past the limit: a graph that does not fit may pay with the wide ones
    const unsigned long long stop_at = V::kTab > kHaloTabMax && most_ids >= 0 ? (unsigned long long)most_ids : ~0ull;
    int dev = 0, sms = 0;
    IRR_CUDA_TRY(cudaGetDevice(&dev));
    IRR_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int64_t tiles = (S + kRunTile - 1) / kRunTile;
    uint8_t *run = nullptr, *cuts = nullptr, *enter = nullptr;
    uint32_t* map = nullptr;
    int32_t *list = nullptr, *tab = nullptr;
    uint16_t *own = nullptr, *place = nullptr;
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
        IRR_CUDA_TRY(alloc_n(&own, n, s));
        IRR_CUDA_TRY(alloc_n(&place, m + 8, s));  // read in whole eights
        IRR_CUDA_TRY(alloc_n(&tab, room, s));
        IRR_CUDA_TRY(cudaMemsetAsync(d_out, 0, sizeof(BuildTotals), s));
        IRR_CUDA_TRY(cudaMemsetAsync(cuts, 0, (size_t)(S > 0 ? S : 1), s));
        if (S > 0) {
            block_runs_kernel<<<(unsigned)std::min<int64_t>(tiles, 8192), kRunTile, 0, s>>>(
                row_off, n, S, (uint32_t)V::kStream, run, map, d_out);
            run_entries_kernel<<<1, 1024, 0, s>>>(map, tiles, enter);
            list_runs_kernel<<<(unsigned)std::min<int64_t>((tiles + 7) / 8, 8192), kRunTile, 0, s>>>(run, enter, S,
                                                                                                    list, d_out);
            cut_runs_kernel<V><<<(unsigned)std::min<int64_t>(S, (int64_t)sms * 128), V::kCutThreads, 0, s>>>(
                src, n, list, run, cut, cuts, own, place, tab, (unsigned long long)room, stop_at, d_out);
            place_items_kernel<false><<<kPlaceCtas, kPlaceThreads, 0, s>>>(n, S, cut, cuts, sums, items, d_out);
            place_items_kernel<true><<<kPlaceCtas, kPlaceThreads, 0, s>>>(n, S, cut, cuts, sums, items, d_out);
            IRR_CUDA_TRY(cudaGetLastError());
        }
        IRR_CUDA_TRY(cudaMemcpyAsync(&got, d_out, sizeof(got), cudaMemcpyDeviceToHost, s));
        IRR_CUDA_TRY(cudaStreamSynchronize(s));
        if (got.flags || got.words > 0xffffffffull || got.ids > 0x7fffffffull) return cudaErrorNotSupported;
        if (most_ids >= 0 && (int64_t)got.ids > most_ids) return cudaErrorNotReady;
        if (got.scratch) return cudaErrorMemoryAllocation;
        out.nwords = (int64_t)got.words;
        out.nids = (int64_t)got.ids;
        out.nitems = got.items;
        IRR_CUDA_TRY(alloc_n(&out.slice_off, S + 1, s));
        IRR_CUDA_TRY(alloc_n(&out.words, out.nwords, s));
        IRR_CUDA_TRY(alloc_n(&out.ids, out.nids, s));
        out.items = items;  // with room for an item per block
        items = nullptr;
        if (S == 0) IRR_CUDA_TRY(cudaMemsetAsync(out.slice_off, 0, sizeof(uint32_t), s));
        if (got.items > 0) {
            // the largest item's entries and 7 on either side, in whole eights (a
            // launch's own argument: the kernel's limit, which all threads share, stays)
            const int smem = (int)((std::min<uint32_t>(got.entries, 2 * V::kStream) + 7 + 15) / 8 * 8 * sizeof(uint16_t));
            static_assert((2 * V::kStream + 22) * sizeof(uint16_t) + 4096 <= 48 * 1024,
                          "with the kernel's own arrays inside the shared memory a launch may have unasked");
            fill_items_kernel<V><<<(unsigned)std::min<int64_t>(got.items, (int64_t)sms * 128), 32 * V::kFillWarps, smem, s>>>(
                row_off, own, place, tab, cut, (int)got.items, out.items, out.slice_off, out.ids, out.words);
            IRR_CUDA_TRY(cudaGetLastError());
        }
        return cudaSuccess;
    };
    const cudaError_t e = go();
    void* tmp[] = {run, cuts, enter, map, list, cut, sums, items, d_out, own, place, tab};
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
        if (p) cudaFreeAsync(p, s);
    *st = Staged{};
}

cudaError_t build_staged(const RowSource& src, int64_t n, int64_t m, bool wide, int64_t most_ids, Staged* st,
                         cudaStream_t s)
{
    free_staged(st, s);
    // Scratch for the tables: a table is at most its item's rows and entries; where
    // all of them are limited, what is beyond need not be held; and where that does
    // not fit, a reuse of 2, then 6, may do (8 and more on MD-like graphs).
    int64_t room = n + m;
    if (most_ids >= 0) room = std::min(room, most_ids);
    for (;;) {
        const cudaError_t e = wide ? build<WideItem>(src, n, m, most_ids, room, st, s)
                                   : build<NarrowItem>(src, n, m, most_ids, room, st, s);
        if (e != cudaErrorMemoryAllocation || room <= m / 6) return e;
        cudaGetLastError();
        room = room > m / 2 ? m / 2 : m / 6;
    }
}

namespace {

// One warp per slice of an item: its rows' ids to their places in col, in the
// slice's order.  A row's picks come before its padding, so pick k of a row is
// an entry for k < its length.
__global__ void __launch_bounds__(32 * kPick) rows_of_items_kernel(const WorkItem* __restrict__ items, int num_items,
                                                                  const uint32_t* __restrict__ slice_off,
                                                                  const uint32_t* __restrict__ words,
                                                                  const int32_t* __restrict__ ids,
                                                                  const uint32_t* __restrict__ row_off,
                                                                  int32_t* __restrict__ col)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int item = blockIdx.x; item < num_items; item += gridDim.x) {
        const WorkItem w = items[item];
        if (8 * warp >= w.nrows) continue;
        const uint32_t o = slice_off[w.row0 / 8 + warp];
        const uint32_t hdr = words[o + lane];
        if (hdr >> 31) continue;  // a padding row
        const uint32_t len = (hdr >> 14) & 1023u;
        const int32_t* tab = ids + w.tab0;
        int32_t* row = col + row_off[w.row0 + ((hdr >> 24) & 127u)];
        for (uint32_t k = lane & 3; k < len; k += 8) {
            const uint32_t pair = words[o + 32 * (k / 8 + 1) + lane];
            row[k] = tab[(pair & 0xffffu) / 16];
            if (k + 4 < len) row[k + 4] = tab[(pair >> 16) / 16];
        }
    }
}

}  // namespace

cudaError_t rows_of_staged(const Staged& st, const WorkItem* items, const uint32_t* row_off, int64_t n, int32_t* col,
                           cudaStream_t s)
{
    if (st.nitems <= 0) return cudaSuccess;
    rows_of_items_kernel<<<(unsigned)std::min<int64_t>(st.nitems, 65536), 32 * kPick, 0, s>>>(
        items, (int)st.nitems, st.slice_off, st.words, st.ids, row_off, col);
    IRR_CUDA_TRY(cudaGetLastError());
    return launch_row_sort(row_off, n, col, s);
}

cudaError_t staged_items_to_host(const WorkItem* d_items, int64_t count, std::vector<WorkItem>* items, cudaStream_t s)
{
    items->resize((size_t)count);
    if (count > 0)
        IRR_CUDA_TRY(cudaMemcpyAsync(items->data(), d_items, sizeof(WorkItem) * (size_t)count, cudaMemcpyDeviceToHost, s));
    return cudaStreamSynchronize(s);
}

}  // namespace irr
