// irr_reduce.cu -- the edge-reduction kernels.
//
// plain_kernel: the reference's per-edge semantics as written -- one thread
//   per edge of the caller's half list, both endpoint contributions added with
//   float4 atomics into a zeroed result.  It replaces compute_gpu
//   (moldyn/irregular/gpu_kernel.cu:21-103), whose shared-memory hash object
//   Sobject (ros.cu:10-68) and global hash Gobject (rog.cu:11-88) become a
//   direct per-node array.
//
// tiled_kernel: owner computes.  The partitioner hands each node a row of
//   directed entries (one per incident edge); a group of G lanes walks the
//   row, evaluates the law for every entry, keeps FP32 partial sums in
//   registers and combines the G partials with error-free TwoSum steps.  Each
//   edge is evaluated from both ends -- the reference duplicates cross-part
//   edges the same way (moldyn/irregular/partitioner.cpp:142-297, paper
//   Sec. II-A) -- so no atomics are needed and every result is bitwise
//   reproducible.  The grid is persistent: CTAs claim node blocks (work
//   items) from a queue, the reference's per-part atomicAdd queue
//   (gpu_kernel.cu:60-77) generalised to (instance, block) items for the
//   batched form.  A block's entries are contiguous, so one bulk (TMA) copy
//   per item moves them into a ring of shared-memory stages a few items
//   ahead of the consumers: the entry stream, which is most of the traffic,
//   is kept in flight while positions are gathered through L1.
//   Entries come in one of two layouts.  CSR rows (consume_item): the rows
//   of a warp start at unrelated offsets, so its reads of the stage collide
//   in shared-memory banks.  Slices (consume_sliced, struct Sliced): the
//   rows of a warp are interleaved and padded, so each step of the warp is
//   one contiguous 256-byte read and the trip count is uniform; with curve-
//   ordered rows whose columns ascend, the lanes of one gather also land on
//   few cache lines.
#include <algorithm>
#include <atomic>
#include <type_traits>
#include <vector>

#include "irr_internal.cuh"

namespace irr {
namespace {

// The atomics bound this kernel: two float4 atomics per edge, 17 bytes of
// atomic traffic for each byte of the list.  Lists are mostly sorted by idx0 (a
// neighbour search writes one node's pairs after another's), so the idx0 side
// of a warp's 32 consecutive edges is summed within each run of equal idx0
// first and added once per run; a warp without a repeated idx0 skips that.
// 300,007 nodes, 9.5 M edges in a random box: 146 -> 97 us, of which the
// idx1 side's gathers and atomics, random over the nodes, are what is left.
template <bool PERIODIC>
__global__ void __launch_bounds__(256) plain_kernel(const float4* __restrict__ pos,
                                                    const int2* __restrict__ edges, int64_t e,
                                                    float4* __restrict__ force, LawParams law)
{
    grid_begin();
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // whole warps walk the list (t0: the warp's first edge)
    for (int64_t t0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); t0 < e; t0 += stride) {
        const bool valid = t0 + lane < e;
        int2 ed = make_int2(-1, -1);
        float fx = 0.f, fy = 0.f, fz = 0.f;
        if (valid) {
            ed = __ldcs(edges + t0 + lane);
            const float4 a = __ldg(pos + ed.x);
            const float4 b = __ldg(pos + ed.y);
            float dx, dy, dz;
            const float s = lj_scalar<PERIODIC>(a, b, law, dx, dy, dz);
            if (s != 0.0f) {  // outside the cutoff otherwise (NaN still propagates)
                fx = __fmul_rn(dx, s);
                fy = __fmul_rn(dy, s);
                fz = __fmul_rn(dz, s);
                atomicAdd(force + ed.y, make_float4(-fx, -fy, -fz, 0.0f));
            }
        }
        const int before = __shfl_up_sync(0xffffffffu, ed.x, 1);
        const bool first = lane == 0 || before != ed.x;  // of a run
        const uint32_t firsts = __ballot_sync(0xffffffffu, first);
        if (firsts != 0xffffffffu) {
            const uint32_t after = firsts & ~((2u << lane) - 1u);
            const int end = after ? __ffs(after) - 1 : 32;  // one past the lane's run
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const float ox = __shfl_down_sync(0xffffffffu, fx, off);
                const float oy = __shfl_down_sync(0xffffffffu, fy, off);
                const float oz = __shfl_down_sync(0xffffffffu, fz, off);
                if (lane + off < end) {
                    fx = __fadd_rn(fx, ox);
                    fy = __fadd_rn(fy, oy);
                    fz = __fadd_rn(fz, oz);
                }
            }
        }
        if (first && valid && !(fx == 0.f && fy == 0.f && fz == 0.f))
            atomicAdd(force + ed.x, make_float4(fx, fy, fz, 0.0f));
    }
}

__global__ void clear_kernel(float4* force, int64_t n)
{
    grid_begin();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        force[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// ---- bulk copy + mbarrier helpers (inline PTX, sm_90+) ----
__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void bulk_load(void* dst_smem, const void* src, uint32_t bytes,
                                          uint64_t* bar)
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_u32(dst_smem)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// One test of phase `parity`; a thread whose phase is not complete may be
// suspended for up to kSuspendNs (it resumes as soon as the phase completes),
// so a waiting warp does not keep issuing polls.
constexpr uint32_t kSuspendNs = 100000;
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity), "r"(kSuspendNs)
        : "memory");
    return done != 0;
}

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for phase `parity` of the barrier; gives up after `limit_ns`
// nanoseconds of wall-clock time (whatever the suspension granted per test).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint64_t limit_ns)
{
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}

// The same bound, polling with a growing sleep (32 ns doubling up to MAX_NS)
// between tests: a warp that waits long -- the producer, waiting for the
// consumers to free a stage -- then takes few issue slots from the warps
// that work on its SM sub-partition (without the sleep a waiting producer
// polled ~450 times per work item).
template <uint32_t MAX_NS>
__device__ __forceinline__ bool mbar_wait_backoff(uint64_t* bar, uint32_t parity, uint64_t limit_ns)
{
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    uint32_t ns = 32;
    for (;;) {
        __nanosleep(ns);
        if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
        if (ns < MAX_NS) ns <<= 1;
    }
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Law parameters the inner loop keeps in registers; the rest (box side as a
// float pair, FP64 cutoff) is read from the instance descriptor on the rare
// paths that need it.
struct HotLaw {
    float half2;   // just under (side/2)^2: rd at or below it never needs a wrap
    float rc2;
    float band;    // |rd - rc2| < band: take the reference's FP64 decision
};

// What the consumers read of an instance.  Batched launches keep it in
// registers across the work items of one instance (its items are
// consecutive); single-instance launches rebuild it from the launch
// parameter for every item, which costs no registers across items.
struct InstHot {
    const float4* __restrict__ pos;
    const uint32_t* __restrict__ row_off;
    const uint32_t* __restrict__ slice_off;
    float4* __restrict__ force;
    const LawParams* __restrict__ cold;
    int64_t n;
    HotLaw H;
};

__device__ __forceinline__ InstHot load_hot(const InstDesc* __restrict__ I)
{
    InstHot h;
    h.pos = I->pos;
    h.row_off = I->row_off;
    h.slice_off = I->slice_off;
    h.force = I->force;
    h.cold = &I->law;
    h.n = I->n;
    h.H.half2 = I->law.half2;
    h.H.rc2 = I->law.rc2;
    h.H.band = I->law.band;
    return h;
}

// Where a launch's consumers find the instance fields (the kernel's last
// parameter, in the constant bank: its fields are read as operands where they
// are used, so they need no registers across items -- at the 56-register
// bound of 4 CTAs x 288 threads that is what removes the spills):
//   SrcGlobal: from the descriptor table in global memory (any batch size);
//   SrcOne:    every item belongs to instance 0, whose descriptor is the
//              parameter;
//   SrcTable:  up to kTableInsts instances, the fields the step loop reads
//              (positions, law constants) of each in the parameter; the
//              per-slice fields, the producer's col / scol and the rare
//              path's law come from the global table.
struct SrcGlobal {
    int unused;
};
struct SrcOne {
    InstDesc d;
};
struct HotEntry {
    const float4* pos;
    HotLaw H;
    float pad;
};
constexpr int kTableInsts = 1024;  // 1024 x 24 B stays inside the 32 KB of kernel parameters
struct SrcTable {
    HotEntry h[kTableInsts];
};

__device__ __forceinline__ InstHot hot_from(const SrcTable& t, const InstDesc* insts, int inst)
{
    const HotEntry& e = t.h[inst];
    const InstDesc* __restrict__ I = insts + inst;
    InstHot h;
    h.pos = e.pos;
    h.row_off = I->row_off;
    h.slice_off = I->slice_off;
    h.force = I->force;
    h.cold = &I->law;
    h.n = I->n;
    h.H = e.H;
    return h;
}

// One component of the minimum image, as b - a: d itself within half the box,
// else the negative of wrap_component (irr_law.cuh), bit for bit -- the larger
// of the two coordinates is taken down by the side first, whichever it is, and
// the sign is d's turned round.
__device__ __forceinline__ float wrap_diff(float a, float b, float d, float half, float shi, float slo)
{
    const float m = __fsub_rn(__fsub_rn(__fsub_rn(fmaxf(a, b), shi), fminf(a, b)), slo);
    return fabsf(d) > half ? (d > 0.f ? m : -m) : d;
}

template <bool PERIODIC>
__device__ __noinline__ bool exact_inside_g(float4 a, float4 b, const LawParams* __restrict__ P)
{
    return exact_inside<PERIODIC>(a, b, *P);
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Two entries (b0, b1) of the row of node a, evaluated with packed FP32x2
// arithmetic (each half rounds exactly as the scalar law in irr_law.cuh), and
// accumulated into the lane's packed partials.  A slot with v == false
// contributes 0 (its b is the row's own position or any valid node).
//
// The differences are formed by scalar subtractions written straight into
// register pairs (the two positions come from separate loads, so a packed
// subtraction would first have to move them into pairs).  They are b - a, the
// law's scalar is -s and the reciprocal -1/rd: every value is the exact
// negative of the scalar law's, and their products are the same bits.
struct PairDiff {
    float2 x, y, z;  // b - a of the two entries
    float2 rd;       // squared distances
};

__device__ __forceinline__ PairDiff pair_diff(float4 a, float4 b0, float4 b1)
{
    PairDiff d;
    d.x = make_float2(__fsub_rn(b0.x, a.x), __fsub_rn(b1.x, a.x));
    d.y = make_float2(__fsub_rn(b0.y, a.y), __fsub_rn(b1.y, a.y));
    d.z = make_float2(__fsub_rn(b0.z, a.z), __fsub_rn(b1.z, a.z));
    d.rd = __ffma2_rn(d.x, d.x, __ffma2_rn(d.y, d.y, __fmul2_rn(d.z, d.z)));
    return d;
}

__device__ __forceinline__ void add_pair(const PairDiff& d, bool in0, bool in1, float2& ax, float2& ay,
                                         float2& az)
{
    float2 r = make_float2(rcp_approx(-d.rd.x), rcp_approx(-d.rd.y));
    const float2 e = __ffma2_rn(d.rd, r, make_float2(1.0f, 1.0f));
    r = __ffma2_rn(r, e, r);             // -rd^-1 (one Newton step)
    const float2 r2 = __fmul2_rn(r, r);  // rd^-2
    float2 s = __fmul2_rn(__fmul2_rn(r2, r2), __ffma2_rn(r2, r, make_float2(0.5f, 0.5f)));
    s.x = in0 ? s.x : 0.0f;
    s.y = in1 ? s.y : 0.0f;
    ax = __ffma2_rn(d.x, s, ax);
    ay = __ffma2_rn(d.y, s, ay);
    az = __ffma2_rn(d.z, s, az);
}

// The rare cases of an entry pair: a pair past half the box (periodic) is
// re-wrapped exactly, and a pair whose rd lies within `band` of the cutoff
// takes the reference's FP64 decision.  Updates d and the in-flags.
template <bool PERIODIC>
__device__ __forceinline__ void rare_pair(float4 a, float4 b0, float4 b1, const HotLaw& H,
                                          const LawParams* __restrict__ cold, PairDiff& d, bool& in0,
                                          bool& in1)
{
    if (PERIODIC && fmaxf(d.rd.x, d.rd.y) > H.half2) {
        // most pairs across the wall cross it on one axis: the others are skipped
        const float half = cold->half, shi = cold->side_hi, slo = cold->side_lo;
        if (fmaxf(fabsf(d.x.x), fabsf(d.x.y)) > half) {
            d.x.x = wrap_diff(a.x, b0.x, d.x.x, half, shi, slo);
            d.x.y = wrap_diff(a.x, b1.x, d.x.y, half, shi, slo);
        }
        if (fmaxf(fabsf(d.y.x), fabsf(d.y.y)) > half) {
            d.y.x = wrap_diff(a.y, b0.y, d.y.x, half, shi, slo);
            d.y.y = wrap_diff(a.y, b1.y, d.y.y, half, shi, slo);
        }
        if (fmaxf(fabsf(d.z.x), fabsf(d.z.y)) > half) {
            d.z.x = wrap_diff(a.z, b0.z, d.z.x, half, shi, slo);
            d.z.y = wrap_diff(a.z, b1.z, d.z.y, half, shi, slo);
        }
        d.rd = __ffma2_rn(d.x, d.x, __ffma2_rn(d.y, d.y, __fmul2_rn(d.z, d.z)));
        in0 = d.rd.x < H.rc2;
        in1 = d.rd.y < H.rc2;
    }
    if (fabsf(__fsub_rn(d.rd.x, H.rc2)) < H.band) in0 = exact_inside_g<PERIODIC>(a, b0, cold);
    if (fabsf(__fsub_rn(d.rd.y, H.rc2)) < H.band) in1 = exact_inside_g<PERIODIC>(a, b1, cold);
}

// A component |d| > side/2 implies rd > (side/2)^2, so the wrap test is one
// compare on rd; it and the cutoff-band test are folded into one branch to
// the rare path (a pair across the box wall, beyond half the box, or within
// 2^-18 of the cutoff).  (A warp vote in front of it measured slower.)
template <bool PERIODIC>
__device__ __forceinline__ void lj_pair(float4 a, float4 b0, float4 b1, bool v0, bool v1, const HotLaw& H,
                                        const LawParams* __restrict__ cold, float2& ax, float2& ay,
                                        float2& az)
{
    PairDiff d = pair_diff(a, b0, b1);
    const float2 t = __fadd2_rn(d.rd, make_float2(-H.rc2, -H.rc2));
    bool rare = fminf(fabsf(t.x), fabsf(t.y)) < H.band;
    if (PERIODIC) rare = rare || fmaxf(d.rd.x, d.rd.y) > H.half2;
    bool in0 = d.rd.x < H.rc2, in1 = d.rd.y < H.rc2;
    if (rare) rare_pair<PERIODIC>(a, b0, b1, H, cold, d, in0, in1);
    add_pair(d, in0 && v0, in1 && v1, ax, ay, az);
}

// The row's result from its G lanes' packed partials: the two halves of each
// lane joined by TwoSum, then the G lanes by a TwoSum butterfly.
//
// The x and y components run as one FP32x2 pair, z as a scalar; every
// operation rounds as its scalar form (a - b is fma(b, -1, a), one rounding),
// so the result is bitwise the scalar TwoSum chain's.
__device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
    return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}

__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2& s, float2& e)
{
    s = __fadd2_rn(a, b);
    const float2 bb = sub2(s, a);
    e = __fadd2_rn(sub2(a, sub2(s, bb)), sub2(b, bb));
}

template <int G>
__device__ __forceinline__ float3 join_partials(float2 ax, float2 ay, float2 az)
{
    float2 h, c;  // (x, y) sums and their carried errors
    float hz, cz;
    two_sum2(make_float2(ax.x, ay.x), make_float2(ax.y, ay.y), h, c);
    two_sum(az.x, az.y, hz, cz);
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) {
        const float2 o = make_float2(__shfl_xor_sync(0xffffffffu, h.x, off, G),
                                     __shfl_xor_sync(0xffffffffu, h.y, off, G));
        const float oz = __shfl_xor_sync(0xffffffffu, hz, off, G);
        const float2 oc = make_float2(__shfl_xor_sync(0xffffffffu, c.x, off, G),
                                      __shfl_xor_sync(0xffffffffu, c.y, off, G));
        const float ocz = __shfl_xor_sync(0xffffffffu, cz, off, G);
        float2 e;
        two_sum2(h, o, h, e);
        c = __fadd2_rn(__fadd2_rn(c, oc), e);
        float ez;
        two_sum(hz, oz, hz, ez);
        cz = __fadd_rn(__fadd_rn(cz, ocz), ez);
    }
    const float2 r = __fadd2_rn(h, c);
    return make_float3(r.x, r.y, __fadd_rn(hz, cz));
}

// join_partials<4>, each lane left with one component: lane 0 x, 1 y, 2 and 3
// z.  The exchanges are arranged so that a lane sums only the components it
// keeps: after the halves, lanes 0 and 1 take x and y over (0, 2) and (1, 3)
// while lanes 2 and 3 take z, then lane 0 x, lane 1 y.  The same pairs are
// added as in join_partials and TwoSum's sum and error do not depend on the
// order of its operands, so the bits are the same, with 6 shuffles instead of
// 12 and one and a half instead of two rounds of sums (halo_kernel at 4M nodes
// 363.4 -> 358.2 us, tiled_kernel at 864,000 atoms 123.8 -> 120.8 us).
__device__ __forceinline__ float join4_scatter(float2 ax, float2 ay, float2 az, int lane)
{
    float2 h, c;
    float hz, cz;
    two_sum2(make_float2(ax.x, ay.x), make_float2(ax.y, ay.y), h, c);
    two_sum(az.x, az.y, hz, cz);
    const bool up = lane & 2;
    const float2 o = make_float2(__shfl_xor_sync(0xffffffffu, up ? h.x : hz, 2, 4),
                                 __shfl_xor_sync(0xffffffffu, h.y, 2, 4));
    const float2 oc = make_float2(__shfl_xor_sync(0xffffffffu, up ? c.x : cz, 2, 4),
                                  __shfl_xor_sync(0xffffffffu, c.y, 2, 4));
    h.x = up ? hz : h.x;
    c.x = up ? cz : c.x;
    float2 e;
    two_sum2(h, o, h, e);
    c = __fadd2_rn(__fadd2_rn(c, oc), e);
    const float p = __shfl_xor_sync(0xffffffffu, lane == 0 ? h.y : h.x, 1, 4);
    const float pc = __shfl_xor_sync(0xffffffffu, lane == 0 ? c.y : c.x, 1, 4);
    const float k = lane == 1 ? h.y : h.x, kc = lane == 1 ? c.y : c.x;
    float s, se;
    two_sum(k, p, s, se);
    return __fadd_rn(s, __fadd_rn(__fadd_rn(kc, pc), se));
}

// Row r's result from its G lanes' partials (valid rows only), written once.
template <int G>
__device__ __forceinline__ void write_row(float4* __restrict__ force, int64_t r, bool valid, float2 ax,
                                          float2 ay, float2 az, int lane)
{
    if constexpr (G == 4) {
        const float f = join4_scatter(ax, ay, az, lane);
        if (valid) reinterpret_cast<float*>(force + r)[lane] = lane == 3 ? 0.f : f;
    } else {
        const float3 f = join_partials<G>(ax, ay, az);
        if (valid && lane == 0) force[r] = make_float4(f.x, f.y, f.z, 0.f);
    }
}

// One row: G lanes; each lane takes entry pairs (k, k + G) with stride 2G.
// Entry k of the row is cols[k - shift].
template <bool PERIODIC, int G>
__device__ __forceinline__ void row_sum(const float4* __restrict__ pos, const int32_t* cols,
                                        uint32_t shift, float4 a, uint32_t beg, uint32_t end, int lane,
                                        const HotLaw& H, const LawParams* __restrict__ cold, float2& ax,
                                        float2& ay, float2& az)
{
    for (uint32_t k = beg + lane; k < end; k += 2 * G) {
        const bool v1 = k + G < end;
        const float4 b0 = __ldg(pos + cols[k - shift]);
        const float4 b1 = v1 ? __ldg(pos + cols[k + G - shift]) : a;
        lj_pair<PERIODIC>(a, b0, b1, true, v1, H, cold, ax, ay, az);
    }
}

constexpr int kConsumerWarps = kConsumerSlices;
constexpr int kPipeThreads = (kConsumerWarps + 1) * 32;

// The rows of one work item that belong to consumer warp `cw`.
template <bool PERIODIC, int G>
__device__ __forceinline__ void consume_item(const WorkItem& w, const InstHot& I,
                                             const int32_t* cols, uint32_t shift, int cw, int lane32)
{
    constexpr int kGroupsPerWarp = 32 / G;
    constexpr int kGroups = kConsumerWarps * kGroupsPerWarp;
    const int lane = lane32 % G;
    const int gid = cw * kGroupsPerWarp + lane32 / G;
    const float4* __restrict__ pos = I.pos;
    const uint32_t* __restrict__ row_off = I.row_off;
    float4* __restrict__ force = I.force;
    const LawParams* __restrict__ cold = I.cold;
    const HotLaw H = I.H;
    const int rounds = (w.nrows + kGroups - 1) / kGroups;
    for (int q = 0; q < rounds; q++) {
        const int rl = q * kGroups + gid;
        const bool valid = rl < w.nrows;
        const int64_t r = (int64_t)w.row0 + rl;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t beg = 0, end = 0;
        if (valid) {
            a = __ldg(pos + r);
            beg = __ldg(row_off + r);
            end = __ldg(row_off + r + 1);
        }
        float2 ax = make_float2(0.f, 0.f), ay = ax, az = ax;
        row_sum<PERIODIC, G>(pos, cols, shift, a, beg, end, lane, H, cold, ax, ay, az);
        write_row<G>(force, r, valid, ax, ay, az, lane);
    }
}

// One lane's entry pair of a slice step, as a single 8-byte load (kept whole
// so the two halves are not split into separately predicated loads).  The
// shared form is volatile: it must stay after the stage's mbarrier wait
// (itself volatile asm), which the compiler could otherwise move it across.
template <bool SHARED>
__device__ __forceinline__ int2 load_pair(const int2* p)
{
    int2 c;
    if (SHARED)
        asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(c.x), "=r"(c.y) : "r"(smem_u32(p)));
    else
        asm("ld.global.nc.v2.b32 {%0, %1}, [%2];" : "=r"(c.x), "=r"(c.y) : "l"(p));
    return c;
}

// The slices of a sliced work item that belong to consumer warp `cw` (one
// slice per warp at a time: lane i*G + l serves row i of the slice).  Word w
// of the instance's sliced array is words[w - shift] (shared memory when
// SHARED).  Each step is one 8-byte load per lane of a contiguous 256-byte
// line; the trip count is the slice's, uniform across the warp, and slots
// past a row's end (padding: the row's own id) are masked.
template <bool PERIODIC, int G, bool SHARED>
__device__ __forceinline__ void consume_sliced(const WorkItem& w, const InstHot& I,
                                               const int32_t* words, uint32_t shift, int cw,
                                               int lane32)
{
    constexpr int R = 32 / G;
    const int lane = lane32 % G;
    const float4* __restrict__ pos = I.pos;
    const uint32_t* __restrict__ row_off = I.row_off;
    const uint32_t* __restrict__ slice_off = I.slice_off;
    float4* __restrict__ force = I.force;
    const LawParams* __restrict__ cold = I.cold;
    const int64_t n = I.n;
    const HotLaw H = I.H;
    const int s0 = w.row0 / R;
    const int ns = (w.nrows + R - 1) / R;
    for (int q = cw; q < ns; q += kConsumerWarps) {
        const uint32_t o0 = __ldg(slice_off + s0 + q);
        const uint32_t steps = (__ldg(slice_off + s0 + q + 1) - o0) >> 6;
        const int64_t r = (int64_t)(s0 + q) * R + lane32 / G;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t len = 0;
        if (r < n) {
            a = __ldg(pos + r);
            len = __ldg(row_off + r + 1) - __ldg(row_off + r);
        }
        const int2* line = reinterpret_cast<const int2*>(words + (o0 - shift)) + lane32;
        float2 ax = make_float2(0.f, 0.f), ay = ax, az = ax;
        // entry 2Gt + lane (+ G) of the row exists for t < n0 (n1)
        const uint32_t n0 = len > (uint32_t)lane ? (len - (uint32_t)lane + 2 * G - 1) / (2 * G) : 0u;
        const uint32_t n1 = len > (uint32_t)(lane + G) ? (len - (uint32_t)lane - G + 2 * G - 1) / (2 * G) : 0u;
        if constexpr (SHARED) {
            // step t's pair at shared address base + 256 t: the masks as
            // bounds on it, no index arithmetic in the loop
            uint32_t sa = smem_u32(line);
            const uint32_t lim0 = sa + 256u * n0, lim1 = sa + 256u * n1, send = sa + 256u * steps;
            for (; sa != send; sa += 256u) {
                int2 c;
                asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(c.x), "=r"(c.y) : "r"(sa));
                const float4 b0 = __ldg(pos + c.x);
                const float4 b1 = __ldg(pos + c.y);
                lj_pair<PERIODIC>(a, b0, b1, sa < lim0, sa < lim1, H, cold, ax, ay, az);
            }
        } else {
            for (uint32_t t = 0; t < steps; t++) {
                const int2 c = load_pair<false>(line + 32 * t);
                const float4 b0 = __ldg(pos + c.x);
                const float4 b1 = __ldg(pos + c.y);
                lj_pair<PERIODIC>(a, b0, b1, t < n0, t < n1, H, cold, ax, ay, az);
            }
        }
        write_row<G>(force, r, r < n, ax, ay, az, lane);
    }
}

// A CTA leaves the queue (one thread of its producer warp, after its last
// claim): the last one to leave clears it for the next launch, so that a step
// needs no clearing launch of its own (3.3 us a step at 864 nodes).
__device__ __forceinline__ void leave_queue(int* queue)
{
    __threadfence();
    if (atomicAdd(queue + 1, 1) == (int)gridDim.x - 1) {
        queue[0] = 0;
        queue[1] = 0;
    }
}

// Persistent owner-computes kernel, warp-specialised.  Warp kConsumerWarps is
// the producer: its lane 0 claims work items from the queue (the next one's
// index and descriptor are read while it waits), and for each item waits until
// its ring stage is empty, publishes the item and
// either bulk-copies the item's entry segment (widened to 16-byte bounds)
// into the stage -- the stage's `full` mbarrier completes on the byte count --
// or, for items read from global memory, just arrives.  The consumer warps
// walk the ring independently: wait `full`, sum their share of the item's
// rows, arrive on `empty` (kConsumerWarps arrivals free the stage).  Waits
// suspend the thread until the phase completes (mbar_try_wait).  Every
// wait is bounded; a wait that gives up sets kStatusWaitTimeout, waits once
// more (bounded) for a copy that may be in flight, and leaves.  wait_ns
// bounds each wait; withhold != 0 (a test of that path) makes every producer
// leave before publishing its first stage, so every consumer's first wait
// runs out and the launch ends with kStatusWaitTimeout and nothing in flight.
//
// Src (SrcGlobal, SrcOne, SrcTable): where the instance fields come from.
enum : int { kStageEnd = 0, kStageGlobal = 1, kStageShared = 2 };
template <bool PERIODIC, int G, class Src>
__global__ void __launch_bounds__(kPipeThreads, kCtasPerSm) tiled_kernel(
    const InstDesc* __restrict__ insts, const WorkItem* __restrict__ items, int num_items,
    int* queue, int* status, int use_stages, uint64_t wait_ns, int withhold,
    const __grid_constant__ Src src)
{
    constexpr bool ONE = std::is_same<Src, SrcOne>::value;
    constexpr bool TABLE = std::is_same<Src, SrcTable>::value;
    extern __shared__ int4 smem_raw[];
    int32_t* stage_base = reinterpret_cast<int32_t*>(smem_raw);
    constexpr int kStageInts = kStageEntries + kColPad;
    __shared__ uint64_t full[kStages];
    __shared__ uint64_t empty[kStages];
    __shared__ WorkItem s_work[kStages];
    __shared__ int s_mode[kStages];
    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kConsumerWarps);
        }
    }
    __syncthreads();
    grid_wait();

    if (warp == kConsumerWarps) {
        if (lane != 0) return;
        if (withhold) {
            leave_queue(queue);
            return;
        }
        int it = (int)blockIdx.x;  // the grid is at most num_items
        WorkItem w = items[it];
        int it1 = (int)gridDim.x + atomicAdd(queue, 1);
        for (int k = 0;; k++) {
            const int s = k % kStages;
            const int use = k / kStages;
            // the next item's descriptor and the claim after it are in flight
            // while this item waits for its stage
            const WorkItem w1 = items[it1 < num_items ? it1 : 0];
            const int it2 = it1 < num_items ? (int)gridDim.x + atomicAdd(queue, 1) : it1;
            if (use > 0 && !mbar_wait_bounded(&empty[s], (uint32_t)(use - 1) & 1u, wait_ns)) {
                atomicOr(status, kStatusWaitTimeout);
                leave_queue(queue);
                return;  // nothing of this stage is in flight: its last copy was consumed
            }
            if (it >= num_items) {
                s_mode[s] = kStageEnd;
                mbar_arrive(&full[s]);
                leave_queue(queue);
                return;
            }
            s_work[s] = w;
            if (use_stages && !(w.flags & kItemDirect)) {
                s_mode[s] = kStageShared;
                const uint32_t a0 = w.ent0 & ~3u;
                const uint32_t words = ((w.ent0 + w.nent - a0) + 3u) & ~3u;
                const InstDesc* I;
                if constexpr (ONE) I = &src.d;
                else I = insts + w.inst;
                const int32_t* ent = (w.flags & kItemSliced) ? I->scol : I->col;
                bulk_load(stage_base + s * kStageInts, ent + a0, words * 4u, &full[s]);
            } else {
                s_mode[s] = kStageGlobal;
                mbar_arrive(&full[s]);
            }
            it = it1;
            w = w1;
            it1 = it2;
        }
    }

    int cur = -1;  // instance whose fields `hot` holds
    InstHot hot{};
    for (int k = 0;; k++) {
        const int s = k % kStages;
        if (!mbar_wait_bounded(&full[s], (uint32_t)(k / kStages) & 1u, wait_ns)) {
            if (lane == 0) atomicOr(status, kStatusWaitTimeout);
            mbar_wait_bounded(&full[s], (uint32_t)(k / kStages) & 1u, wait_ns);
            return;
        }
        const int mode = s_mode[s];
        if (mode == kStageEnd) return;
        const WorkItem w = s_work[s];
        const InstDesc* I;
        if constexpr (ONE) {
            I = &src.d;
            hot = load_hot(I);
        } else if constexpr (TABLE) {
            I = insts + w.inst;
            hot = hot_from(src, insts, w.inst);
        } else {
            I = insts + w.inst;
            if (w.inst != cur) {
                hot = load_hot(I);
                cur = w.inst;
            }
        }
        if (w.flags & kItemSliced) {
            if (mode == kStageShared)
                consume_sliced<PERIODIC, G, true>(w, hot, stage_base + s * kStageInts, w.ent0, warp,
                                                  lane);
            else
                consume_sliced<PERIODIC, G, false>(w, hot, I->scol, 0u, warp, lane);
        } else if (mode == kStageShared) {
            consume_item<PERIODIC, G>(w, hot, stage_base + s * kStageInts, w.ent0 & ~3u, warp, lane);
        } else {
            consume_item<PERIODIC, G>(w, hot, I->col, 0u, warp, lane);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
    }
}

// ---- staged ("halo") layout: positions staged in shared memory ----
//
// halo_kernel: the same persistent, warp-specialised owner-computes reduction
// over the staged layout (irr_staged.cu).  Per work item the producer warp
// bulk-copies the item's words (headers and 16-bit table offsets) into shared
// memory, and its 32 lanes gather the item's table -- the positions of every
// node its rows touch, ~465 for 64 rows -- behind them with 16-byte cp.async
// copies; the item's `full` barrier completes when the bulk copy's bytes and
// all 32 lanes' copies have landed (1 + 32 arrivals).  The consumers read each
// entry's position from shared memory (a 128-bit load at a table offset), so
// the law's operands arrive in tens of cycles instead of an L1 miss's
// hundreds, and the entry order of the layout spreads each quarter-warp's 8
// loads over the 8 bank groups.  G = 4 lanes per row.
//
// What bounds it: the issue slots of the law (83 % of the time with an
// instant producer) and the refill of the stages, so the items lie in one ring
// buffer, each taking the bytes it needs (~17 KB of the 24 KB limit at 64
// neighbours per node) in whole 128-byte lines, up to kHaloSlots of them: three
// fit where two stages of the limit's size did.  Everything else an item needs
// (its table ids, descriptor, claim) goes through the producer's registers,
// read one or two items ahead, so that the ring gets all of the shared memory
// of a quarter SM.  4,194,304 nodes, 64 neighbours: 367.8 us with two stages
// of 24 KB, 368.8 with a ring of 49,152 bytes, 358.6 with this one; 48 systems
// of 2,000 to 120,000 nodes in one launch 153.5 -> 139.5 us, 65,536 nodes with
// 32 neighbours 10.6 -> 9.9 us.
constexpr int kHaloRingBytes = 56064;
constexpr int kHaloSlots = 4;
// The consumers add a table's address to both 16-bit halves of a word at once,
// and a slot's two addresses share a word, which needs every shared address of
// the CTA below 2^16: the ring, the barriers, the metadata and the system's
// reserved kilobyte.
static_assert(kHaloRingBytes >= 4 * kHaloStreamMax + 16 * kHaloTabMax &&
                  kHaloRingBytes >= 4 * kHaloWideStreamMax + 16 * kHaloWideTabMax && kHaloRingBytes % 128 == 0 &&
                  kHaloRingBytes + 1024 + 1024 < 65536,
              "an item fits the ring, shared addresses fit 16 bits");
static_assert(8 * kHaloSlicesPerItem <= 64, "a row's index in its item fits the header's 6 bits");

__device__ __forceinline__ void cp_async16(uint32_t dst_smem, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}

// One arrival on `bar` once every cp.async this thread issued before has
// landed (noinc: the barrier's expected count includes it).
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Shared loads kept after the item's barrier wait (volatile, like load_pair).
__device__ __forceinline__ uint32_t lds32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

__device__ __forceinline__ float4 lds128(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr));
    return v;
}

// Longest sleep between two tests of a barrier, ns (32 / 64 to 512 / 512: no
// difference).
constexpr uint32_t kConsumerSleep = 128, kProducerSleep = 256;

// The two neighbours of a lane's step: one word of two 16-bit table byte
// offsets, then the two positions from the table.
__device__ __forceinline__ void halo_operands(uint32_t addr, uint32_t tab_pair, float4& b0, float4& b1)
{
    const uint32_t wd = lds32(addr) + tab_pair;
    b0 = lds128(wd & 0xffffu);
    b1 = lds128(wd >> 16);
}

// One slice: lane i * 4 + l of the warp serves row i.  addr: this lane's
// header word; steps: words per lane after it.
struct HaloSlice {
    uint32_t addr;
    uint32_t steps;
    uint32_t tab_pair;  // the table's address in both halves
    int row0;
};

template <bool PERIODIC>
__device__ __forceinline__ void halo_slice(const HaloSlice& sl, const InstHot& I)
{
    const int lane = threadIdx.x & 3;
    const HotLaw H = I.H;
    uint32_t addr = sl.addr;
    // header: own byte offset | len << 14 | row-in-item << 24 (1 << 31: padding)
    const uint32_t hdr = lds32(addr);
    const float4 a = lds128((sl.tab_pair & 0xffffu) + (hdr & 0x3fffu));
    const uint32_t len = (hdr >> 14) & 0x3ffu;
    float2 ax = make_float2(0.f, 0.f), ay = ax, az = ax;
    // entry 8t + lane (+ 4) of the row exists for 8t < len - lane (- 4): as
    // bounds on step t's word address, base + 128 (t + 1)
    const uint32_t lim0 = addr + 16u * ((len + 7u - (uint32_t)lane) & ~7u);
    const uint32_t lim1 = addr + 16u * ((len + 3u - (uint32_t)lane) & ~7u);
    const uint32_t end = addr + 128u * sl.steps;
    for (; addr != end;) {
        addr += 128u;
        float4 b0, b1;
        halo_operands(addr, sl.tab_pair, b0, b1);
        lj_pair<PERIODIC>(a, b0, b1, addr <= lim0, addr <= lim1, H, I.cold, ax, ay, az);
    }
    write_row<4>(I.force, (int64_t)sl.row0 + ((hdr >> 24) & 0x3fu), !(hdr >> 31), ax, ay, az, lane);
}

// WIDE: items to the wide limits, each up to two thirds of the ring, beside which
// much of the next one loads.  Its table's ids are too many for the producer's
// registers and are read when there is room for them, so ids and positions are
// one chain, and that, not issue, bounds it: 262,144 nodes with 248 neighbours
// issue in 48 % of the active cycles (narrow items at 64 neighbours: 77 %).
template <bool PERIODIC, bool WIDE, class Src>
__global__ void __launch_bounds__(kPipeThreads, kCtasPerSm) halo_kernel(
    const InstDesc* __restrict__ insts, const WorkItem* __restrict__ items, int num_items,
    int* queue, int* status, uint64_t wait_ns, int withhold, const __grid_constant__ Src src)
{
    constexpr bool ONE = std::is_same<Src, SrcOne>::value;
    constexpr bool TABLE = std::is_same<Src, SrcTable>::value;
    extern __shared__ __align__(128) unsigned char ring[];
    __shared__ uint64_t full[kHaloSlots];
    __shared__ uint64_t empty[kHaloSlots];
    // per slot: (instance, first row, slices -- 0: no more items, ring offset |
    // table address << 16), and its slices (byte offset | steps << 16), so
    // that the consumers read no global memory
    __shared__ __align__(16) int4 s_meta[kHaloSlots];
    __shared__ uint32_t s_slice[kHaloSlots][kHaloSlicesPerItem];
    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kHaloSlots; s++) {
            mbar_init(&full[s], 33);  // the bulk copy's arrive + one per producer lane
            mbar_init(&empty[s], kConsumerWarps);
        }
    }
    __syncthreads();
    grid_wait();

    if (warp == kConsumerWarps) {
        if (withhold) {
            if (queue && lane == 0) leave_queue(queue);
            return;
        }
        // The chain from a claim to an item's positions is four dependent trips
        // to memory (queue, descriptor, table ids, positions), ~3 us in a row,
        // nearly as long as the consumers take over an item.  So it is spread
        // over the iterations before: in iteration k, item k's positions are
        // copied, item k + 1's table ids (20 to a lane) and slice offsets (lane
        // j holds the j-th) are read into registers, item k + 2 is claimed and
        // its descriptor is read.  An index of num_items or more: no more work.
        auto claim = [&](int last) {
            if (!queue) return last + (int)gridDim.x;
            return lane == 0 ? (int)gridDim.x + atomicAdd(queue, 1) : 0;
        };
        auto describe = [&](int& it) {
            if (queue) it = __shfl_sync(0xffffffffu, it, 0);
            return items[it < num_items ? it : 0];
        };
        constexpr int kIds = WIDE ? 1 : (kHaloTabMax + 31) / 32;
        int32_t ids[kIds];
        uint32_t so = 0;
        auto fetch = [&](const WorkItem& w) {
            const InstDesc* I;
            if constexpr (ONE) I = &src.d;
            else I = insts + w.inst;
            if constexpr (!WIDE) {
                const int32_t* __restrict__ tab = I->tab + w.tab0 + lane;
#pragma unroll
                for (int j = 0; j < kIds; j++)
                    if (32 * j + lane < (int)w.ntab) ids[j] = __ldg(tab + 32 * j);
            }
            if (lane <= (w.nrows + 7) / 8) so = __ldg(I->slice_off + w.row0 / 8 + lane) - w.ent0;
        };
        int it = (int)blockIdx.x, it1 = claim(it);  // the grid is at most num_items
        WorkItem w = items[it];
        fetch(w);
        WorkItem w1 = describe(it1);
        const uint32_t ring0 = smem_u32(ring);
        uint32_t head = 0;   // ring offset after the newest item
        int live = 0;        // oldest item whose slot is not known to be free
        for (int k = 0;; k++) {
            const int s = k % kHaloSlots;
            const bool more = it < num_items;
            int it2 = claim(it1);
            // whole 128-byte lines, so that every item starts on one
            const uint32_t size = more ? (4u * w.nent + 16u * w.ntab + 127u) & ~127u : 0u;
            // room for the item: a free slot, and `size` bytes after the newest
            // item or, wrapped, at the ring's start; else the oldest item's end
            // is waited for
            for (;;) {
                if (live == k) {
                    head = 0;
                    break;
                }
                if (k - live < kHaloSlots) {
                    const uint32_t tail = ((uint32_t)s_meta[live % kHaloSlots].w & 0xffffu) - ring0;
                    if (head > tail) {
                        if (size <= (uint32_t)kHaloRingBytes - head) break;
                        if (size <= tail) {
                            head = 0;
                            break;
                        }
                    } else if (size <= tail - head) {
                        break;
                    }
                }
                int ok = 1;
                if (lane == 0)
                    ok = mbar_wait_backoff<kProducerSleep>(&empty[live % kHaloSlots],
                                                           (uint32_t)(live / kHaloSlots) & 1u, wait_ns)
                             ? 1
                             : 0;
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) {  // a wait gave up: leave with none of this lane's copies in flight
                    if (lane == 0) {
                        atomicOr(status, kStatusWaitTimeout);
                        if (queue) leave_queue(queue);
                    }
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    return;
                }
                live++;
            }
            if (!more) {  // no more work: complete the slot's phase for the consumers
                if (lane == 0) {
                    s_meta[s] = make_int4(0, 0, 0, 0);
                    mbar_arrive(&full[s]);
                    if (queue) leave_queue(queue);
                }
                mbar_arrive(&full[s]);
                asm volatile("cp.async.wait_all;" ::: "memory");
                return;
            }
            const InstDesc* I;
            if constexpr (ONE) I = &src.d;
            else I = insts + w.inst;
            const uint32_t base = ring0 + head, tab = base + 4u * w.nent;
            const int ns = (w.nrows + 7) / 8;
            // the metadata, written before the item is published: lane 0's
            // arrive (release) follows every lane's writes through __syncwarp
            const uint32_t next = __shfl_down_sync(0xffffffffu, so, 1);
            if (lane < ns) s_slice[s][lane] = 4u * so | ((((next - so) >> 5) - 1u) << 16);
            if (lane == 0) s_meta[s] = make_int4(w.inst, w.row0, ns, (int)(base | (tab << 16)));
            __syncwarp();
            if (lane == 0) bulk_load(ring + head, I->words + w.ent0, w.nent * 4u, &full[s]);
            const float4* __restrict__ pos = I->pos;
            if constexpr (WIDE) {
                const int32_t* __restrict__ src_ids = I->tab + w.tab0;
#pragma unroll 8
                for (uint32_t j = lane; j < w.ntab; j += 32) cp_async16(tab + 16u * j, pos + __ldg(src_ids + j));
            } else {
#pragma unroll
                for (int j = 0; j < kIds; j++)
                    if (32 * j + lane < (int)w.ntab) cp_async16(tab + 512u * j + 16u * lane, pos + ids[j]);
            }
            cp_async_arrive(&full[s]);
            head += size;
            it = it1;
            w = w1;
            if (it < num_items) fetch(w);
            it1 = it2;
            w1 = describe(it1);
        }
    }

    int cur = -1;
    InstHot hot{};
    for (int k = 0;; k++) {
        const int s = k % kHaloSlots;
        if (!mbar_wait_backoff<kConsumerSleep>(&full[s], (uint32_t)(k / kHaloSlots) & 1u, wait_ns)) {
            if (lane == 0) atomicOr(status, kStatusWaitTimeout);
            mbar_wait_backoff<kConsumerSleep>(&full[s], (uint32_t)(k / kHaloSlots) & 1u, wait_ns);
            return;
        }
        const int4 m = s_meta[s];
        if (m.z == 0) return;
        if constexpr (ONE) {
            hot = load_hot(&src.d);
        } else if constexpr (TABLE) {
            hot = hot_from(src, insts, m.x);
        } else if (m.x != cur) {
            hot = load_hot(insts + m.x);
            cur = m.x;
        }
        // warp w takes slice (w + k) mod 8 of the CTA's k-th item: slice 0
        // holds an item's longest rows, so a fixed assignment would always give
        // one warp the longest slice
        for (int q = (warp + k) % kConsumerWarps; q < m.z; q += kConsumerWarps) {
            const uint32_t sl = s_slice[s][q], w = (uint32_t)m.w;
            halo_slice<PERIODIC>(HaloSlice{(w & 0xffffu) + (sl & 0xffffu) + 4u * (uint32_t)lane, sl >> 16,
                                           (w >> 16) * 0x10001u, m.y},
                                 hot);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
    }
}

// A kernel's shared-memory limit, set once per device (2 us a call).
class DeviceOnce {
public:
    cudaError_t max_shared(const void* kern, int bytes)
    {
        int dev = 0;
        IRR_CUDA_TRY(cudaGetDevice(&dev));
        const bool known = dev >= 0 && dev < 64;
        const uint64_t bit = known ? 1ull << dev : 0;
        if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
        IRR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        done_.fetch_or(bit, std::memory_order_release);
        return cudaSuccess;
    }

private:
    std::atomic<uint64_t> done_{0};
};

template <bool PERIODIC, bool WIDE, class Src>
cudaError_t launch_halo_src(const InstDesc* d_insts, const WorkItem* d_items, int num_items,
                            int* d_queue, int grid, int* d_status, cudaStream_t s, const Src& src,
                            const WaitPolicy& wp)
{
    auto kern = halo_kernel<PERIODIC, WIDE, Src>;
    static DeviceOnce once;
    IRR_CUDA_TRY(once.max_shared(reinterpret_cast<const void*>(kern), kHaloRingBytes));
    if (grid <= 0 || num_items <= 0) return cudaSuccess;
    // claims run two items ahead of a CTA's positions, which with a few items
    // per CTA leaves some with three and others with one: up to 4 items per CTA
    // they are dealt out in turn.  Claimed and dealt, us at 64 neighbours: 1 item
    // per CTA 8.9 and 8.6, 1.5 13.6 and 10.9, 2.5 18.0 and 14.5, 3.5 21.5 and
    // 19.5, 4 22.4 and 22.3, 5 26.8 and 24.5, 6 29.8 and 29.7, 8 36.3 and 38.1, 16
    // 63.8 and 69.6, 108 386 and 429; at 32 neighbours they cross at 6 too.
    int* const queue = num_items <= 4 * grid ? nullptr : d_queue;
    return launch_chained(kern, (unsigned)std::min(grid, num_items), kPipeThreads, kHaloRingBytes, s, d_insts,
                          d_items, num_items, queue, d_status, wp.wait_ns, wp.withhold, src);
}

template <bool PERIODIC, bool WIDE>
cudaError_t launch_halo_p(const InstDesc* d_insts, const WorkItem* d_items, int num_items,
                          int* d_queue, int grid, int* d_status, cudaStream_t s,
                          const InstDesc* host_insts, int num_insts, const WaitPolicy& wp)
{
    if (host_insts && num_insts == 1)
        return launch_halo_src<PERIODIC, WIDE>(d_insts, d_items, num_items, d_queue, grid, d_status, s,
                                         SrcOne{host_insts[0]}, wp);
    if (host_insts && num_insts > 1 && num_insts <= kTableInsts) {
        static thread_local SrcTable t;
        for (int k = 0; k < num_insts; k++) {
            const InstDesc& d = host_insts[k];
            t.h[k] = HotEntry{d.pos, HotLaw{d.law.half2, d.law.rc2, d.law.band}, 0.f};
        }
        return launch_halo_src<PERIODIC, WIDE>(d_insts, d_items, num_items, d_queue, grid, d_status, s, t,
                                         wp);
    }
    return launch_halo_src<PERIODIC, WIDE>(d_insts, d_items, num_items, d_queue, grid, d_status, s,
                                     SrcGlobal{0}, wp);
}

template <bool PERIODIC, int G, class Src>
cudaError_t launch_tiled_src(const TiledShape& shape, const InstDesc* d_insts,
                             const WorkItem* d_items, int num_items, int* d_queue, int grid,
                             int* d_status, cudaStream_t s, const Src& src, const WaitPolicy& wp)
{
    auto kern = tiled_kernel<PERIODIC, G, Src>;
    const size_t smem =
        shape.stage_smem ? (size_t)kStages * (kStageEntries + kColPad) * sizeof(int32_t) : 0;
    static DeviceOnce once;
    if (smem > 48 * 1024) IRR_CUDA_TRY(once.max_shared(reinterpret_cast<const void*>(kern), (int)smem));
    if (grid <= 0 || num_items <= 0) return cudaSuccess;
    return launch_chained(kern, (unsigned)std::min(grid, num_items), kPipeThreads, smem, s, d_insts, d_items,
                          num_items, d_queue, d_status, shape.stage_smem, wp.wait_ns, wp.withhold, src);
}

template <bool PERIODIC, int G>
cudaError_t launch_tiled_g(const TiledShape& shape, const InstDesc* d_insts,
                           const WorkItem* d_items, int num_items, int* d_queue, int grid,
                           int* d_status, cudaStream_t s, const InstDesc* host_insts,
                           int num_insts, const WaitPolicy& wp)
{
    if (host_insts && num_insts == 1)
        return launch_tiled_src<PERIODIC, G>(shape, d_insts, d_items, num_items, d_queue, grid,
                                             d_status, s, SrcOne{host_insts[0]}, wp);
    if (host_insts && num_insts > 1 && num_insts <= kTableInsts) {
        static thread_local SrcTable t;  // 28 KB: kept off the stack
        for (int k = 0; k < num_insts; k++) {
            const InstDesc& d = host_insts[k];
            t.h[k] = HotEntry{d.pos, HotLaw{d.law.half2, d.law.rc2, d.law.band}, 0.f};
        }
        return launch_tiled_src<PERIODIC, G>(shape, d_insts, d_items, num_items, d_queue, grid,
                                             d_status, s, t, wp);
    }
    return launch_tiled_src<PERIODIC, G>(shape, d_insts, d_items, num_items, d_queue, grid,
                                         d_status, s, SrcGlobal{0}, wp);
}

template <bool PERIODIC>
cudaError_t launch_tiled_p(const TiledShape& sh, const InstDesc* a, const WorkItem* b, int n,
                           int* q, int grid, int* st, cudaStream_t s, const InstDesc* hi, int ni,
                           const WaitPolicy& wp)
{
    switch (sh.lanes_per_row) {
    case 1: return launch_tiled_g<PERIODIC, 1>(sh, a, b, n, q, grid, st, s, hi, ni, wp);
    case 2: return launch_tiled_g<PERIODIC, 2>(sh, a, b, n, q, grid, st, s, hi, ni, wp);
    case 4: return launch_tiled_g<PERIODIC, 4>(sh, a, b, n, q, grid, st, s, hi, ni, wp);
    case 8: return launch_tiled_g<PERIODIC, 8>(sh, a, b, n, q, grid, st, s, hi, ni, wp);
    case 16: return launch_tiled_g<PERIODIC, 16>(sh, a, b, n, q, grid, st, s, hi, ni, wp);
    case 32: return launch_tiled_g<PERIODIC, 32>(sh, a, b, n, q, grid, st, s, hi, ni, wp);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t launch_plain(const float4* pos, const int2* edges, int64_t e, float4* force, int64_t n,
                         const LawParams& law, int sms, cudaStream_t s)
{
    if (n > 0)
        IRR_CUDA_TRY(launch_chained(clear_kernel, (unsigned)std::min<int64_t>((n + 255) / 256, (int64_t)sms * 8), 256, 0,
                                    s, force, n));
    if (e <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)std::min<int64_t>((e + 255) / 256, (int64_t)sms * 32);
    return law.periodic ? launch_chained(plain_kernel<true>, grid, 256, 0, s, pos, edges, e, force, law)
                        : launch_chained(plain_kernel<false>, grid, 256, 0, s, pos, edges, e, force, law);
}

cudaError_t launch_tiled(const TiledShape& shape, const InstDesc* d_insts,
                         const WorkItem* d_items, int num_items, int* d_queue, int grid,
                         int* d_status, cudaStream_t s, const InstDesc* host_insts, int num_insts,
                         const WaitPolicy& wp)
{
    if (!d_queue) return cudaErrorInvalidValue;
    if (shape.staged) {
        if (shape.lanes_per_row != 4) return cudaErrorInvalidValue;
        auto launch = shape.staged == 2 ? (shape.periodic ? launch_halo_p<true, true> : launch_halo_p<false, true>)
                                        : (shape.periodic ? launch_halo_p<true, false> : launch_halo_p<false, false>);
        return launch(d_insts, d_items, num_items, d_queue, grid, d_status, s, host_insts, num_insts, wp);
    }
    return shape.periodic ? launch_tiled_p<true>(shape, d_insts, d_items, num_items, d_queue, grid,
                                                 d_status, s, host_insts, num_insts, wp)
                          : launch_tiled_p<false>(shape, d_insts, d_items, num_items, d_queue,
                                                  grid, d_status, s, host_insts, num_insts, wp);
}

void make_work_items(const uint32_t* row_off, int64_t n, int inst, int max_rows, int staged,
                     std::vector<WorkItem>& out, int round_rows)
{
    int64_t r = 0;
    while (r < n) {
        WorkItem w{};
        w.inst = inst;
        w.row0 = (int32_t)r;
        w.ent0 = row_off[r];
        int64_t q = r + 1;
        if ((int64_t)(row_off[q] - row_off[r]) > kStageEntries) {
            w.flags = kItemDirect;  // one long row: read from global memory
        } else {
            while (q < n && q - r < max_rows && (int64_t)(row_off[q + 1] - row_off[r]) <= kStageEntries)
                q++;
            if (q < n && q - r > round_rows) q = r + (q - r) / round_rows * round_rows;
        }
        w.nrows = (int32_t)(q - r);
        w.nent = row_off[q] - row_off[r];
        if (!staged || w.nent == 0) w.flags |= kItemDirect;
        out.push_back(w);
        r = q;
    }
}

void make_instance_items(const uint32_t* host_row_off, const Sliced& sl, int64_t n, int inst,
                         const TiledShape& shape, std::vector<WorkItem>& out)
{
    if (sl.lanes != 0 && sl.lanes == shape.lanes_per_row)
        make_sliced_items(sl, n, inst, shape.block_nodes, shape.stage_smem, out);
    else
        make_work_items(host_row_off, n, inst, shape.block_nodes, shape.stage_smem, out,
                        kConsumerSlices * (32 / shape.lanes_per_row));
}

void make_sliced_items(const Sliced& sl, int64_t n, int inst, int max_rows, int staged,
                       std::vector<WorkItem>& out)
{
    const int R = 32 / sl.lanes;
    const int64_t max_slices = std::max<int64_t>(1, max_rows / R);
    const uint32_t* off = sl.host_off.data();
    int64_t q = 0;
    while (q < sl.slices) {
        int64_t e = q + 1;
        if ((int64_t)(off[e] - off[q]) <= kStageEntries) {
            while (e < sl.slices && e - q < max_slices &&
                   (int64_t)(off[e + 1] - off[q]) <= kStageEntries)
                e++;
            // whole rounds of the consumer warps where the item allows it
            if (e < sl.slices && e - q > kConsumerSlices) e = q + (e - q) / kConsumerSlices * kConsumerSlices;
        }
        WorkItem w{};
        w.inst = inst;
        w.row0 = (int32_t)(q * R);
        w.nrows = (int32_t)(std::min<int64_t>(n, e * R) - q * R);
        w.ent0 = off[q];
        w.nent = off[e] - off[q];
        w.flags = kItemSliced;
        if (!staged || w.nent == 0 || (int64_t)w.nent > kStageEntries) w.flags |= kItemDirect;
        out.push_back(w);
        q = e;
    }
}

}  // namespace irr
