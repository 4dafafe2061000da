// irr_md.cuh -- the MD object, shared with the serving loop.
#pragma once
#include <string>
#include <vector>

#include "irr_internal.cuh"
#include "../../include/irregular_gb300.h"

using irr::InstDesc;
using irr::LawParams;
using irr::PartitionOut;
using irr::TiledShape;
using irr::WorkItem;

// ---- the integrator, per atom (shared by the per-system kernels of
// irr_md.cu and the batched ones of the serving loop, so a system's
// trajectory does not depend on which of them ran it)

// x into [0, L).  An atom moves much less than a box per step, so one shift
// of +-L covers the step (FP64 division is slow here); the floor form is the
// fallback and gives the same value for x in [-L, 2L).
// (Not inlined: the compiler computes 2 L and -L ahead, in FP64, for atoms that
// need neither.)
static __device__ __noinline__ double md_wrap_box(double x, double L)
{
    if (x >= L) {
        x = x < 2.0 * L ? x - L : x - L * floor(x / L);
    } else if (x < 0.0) {
        x = x >= -L ? x + L : x - L * floor(x / L);
    }
    if (x >= L) x -= L;  // x = -tiny rounds up to L
    if (x < 0.0) x = 0.0;
    return x;
}

// +0 <= x < L by integer compares of the bit patterns (for x with the sign bit
// clear the IEEE order is the integer order): md_wrap_box(x, L) is x.  By the
// upper words alone: a value within 2^-20 of L may be called outside.
__device__ __forceinline__ bool md_inside(double x, double L)
{
    return (uint32_t)__double2hiint(x) < (uint32_t)__double2hiint(L);
}

// md_wrap_box by one addition where that brings x inside, which leaves out the
// far, the rounded (x = -tiny) and the signed zero.
__device__ __forceinline__ double md_wrap_near(double x, double L)
{
    if (md_inside(x, L)) return x;
    const int flip = ~__double2hiint(x) & (int)0x80000000;  // x + L below 0, x - L above
    const double y = x + __hiloint2double(__double2hiint(L) ^ flip, __double2loint(L));
    return md_inside(y, L) ? y : md_wrap_box(x, L);
}

// A float and a double at one another's precision by integer arithmetic, the
// conversion instructions' values: those run at the FP64 rate, which bounds the
// integrator.  ok: a normal float (or a positive double that becomes one);
// others take the instruction.
__device__ __forceinline__ bool md_widens(float f)
{
    const uint32_t e = __float_as_uint(f) & 0x7f800000u;
    return e != 0 && e != 0x7f800000u;
}
__device__ __forceinline__ double md_widen(float f)
{
    const uint32_t u = __float_as_uint(f);
    return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(u << 29));
}
__device__ __forceinline__ bool md_narrows(double d)  // exponents 897 to 1150, sign clear
{
    return (uint32_t)(__double2hiint(d) >> 20) - 897u <= 253u;
}
__device__ __forceinline__ float md_narrow(double d)
{
    const uint32_t lo = (uint32_t)__double2loint(d), left = lo << 3;  // what is rounded away
    const uint32_t f = __funnelshift_l(lo, (uint32_t)__double2hiint(d), 3) - 0xc0000000u;
    return __uint_as_float(f + ((left | (f & 1u)) > 0x80000000u ? 1u : 0u));  // to nearest, ties to even
}
// Three at a time.  The instructions are out of line: in line the compiler
// predicates them, and one that is predicated off still takes its turn.
static __device__ __noinline__ double md_widen_any(float f) { return (double)f; }
static __device__ __noinline__ float md_narrow_any(double d) { return (float)d; }
__device__ __forceinline__ void md_widen3(float4 f, double& x, double& y, double& z)
{
    if (md_widens(f.x) && md_widens(f.y) && md_widens(f.z)) {
        x = md_widen(f.x);
        y = md_widen(f.y);
        z = md_widen(f.z);
    } else {
        x = md_widen_any(f.x);
        y = md_widen_any(f.y);
        z = md_widen_any(f.z);
    }
}
__device__ __forceinline__ void md_narrow3(double x, double y, double z, float& fx, float& fy, float& fz)
{
    if (md_narrows(x) && md_narrows(y) && md_narrows(z)) {
        fx = md_narrow(x);
        fy = md_narrow(y);
        fz = md_narrow(z);
    } else {
        fx = md_narrow_any(x);
        fy = md_narrow_any(y);
        fz = md_narrow_any(z);
    }
}

// What bounds the integrator: FP64 issue (16 SM cycles a warp instruction on
// this part) until only the 9 multiply-adds are left of it, then HBM.  864,000
// atoms: 33.1 -> 19.3 us a step, 5.7 TB/s of its 128 bytes an atom, the
// conversions and what the compiler ran ahead of the wrap having been the rest.
// Atom i: KICKS half kicks v += dt/2 * 48 f (KICKS = 2 fuses the closing
// kick of the step before, with the same forces: each kick rounds as a
// separate one would), then the drift x += dt v wrapped into [0, L), and the
// float copy for the reduction (a value that rounds up to L wraps to 0).
// hk: md_half_kick(dt).
inline double md_half_kick(double dt) { return 0.5 * dt * 48.0; }

template <int KICKS>
__device__ __forceinline__ void md_kick_drift_atom(double* __restrict__ x, double* __restrict__ v,
                                                   const float4* __restrict__ f, int64_t i,
                                                   double dt, double hk, double L, float Lf,
                                                   float4* __restrict__ pos4)
{
    const float4 fi = f[i];
    double* xi = x + 3 * i;
    double* vi = v + 3 * i;
    double gx, gy, gz;
    md_widen3(fi, gx, gy, gz);
    double vx = vi[0], vy = vi[1], vz = vi[2];
#pragma unroll
    for (int k = 0; k < KICKS; k++) {
        vx = __fma_rn(hk, gx, vx);
        vy = __fma_rn(hk, gy, vy);
        vz = __fma_rn(hk, gz, vz);
    }
    double px = __fma_rn(dt, vx, xi[0]);
    double py = __fma_rn(dt, vy, xi[1]);
    double pz = __fma_rn(dt, vz, xi[2]);
    // a branch for the warp: per atom the compiler ran the wrap's FP64
    // instructions, predicated off, for every atom
    if (__any_sync(__activemask(), !(md_inside(px, L) && md_inside(py, L) && md_inside(pz, L)))) {
        px = md_wrap_near(px, L);
        py = md_wrap_near(py, L);
        pz = md_wrap_near(pz, L);
    }
    vi[0] = vx;
    vi[1] = vy;
    vi[2] = vz;
    xi[0] = px;
    xi[1] = py;
    xi[2] = pz;
    float fx, fy, fz;
    md_narrow3(px, py, pz, fx, fy, fz);
    if (fx >= Lf) fx = 0.f;
    if (fy >= Lf) fy = 0.f;
    if (fz >= Lf) fz = 0.f;
    pos4[i] = make_float4(fx, fy, fz, 0.f);
}

// Atom i: the closing half kick of a step.
__device__ __forceinline__ void md_kick_atom(double* __restrict__ v, const float4* __restrict__ f,
                                             int64_t i, double hk)
{
    const float4 fi = f[i];
    double* vi = v + 3 * i;
    double gx, gy, gz;
    md_widen3(fi, gx, gy, gz);
    vi[0] = __fma_rn(hk, gx, vi[0]);
    vi[1] = __fma_rn(hk, gy, vi[1]);
    vi[2] = __fma_rn(hk, gz, vi[2]);
}

struct irr_md {
    irr_md_config cfg{};
    int device = 0;
    int sms = 0;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    std::string err;
    int64_t n = 0;
    LawParams law{};
    TiledShape shape{};
    double* x = nullptr;       // [3n] positions, execution order
    double* v = nullptr;       // [3n] velocities
    double* tmp = nullptr;     // [3n] permutation scratch
    float4* pos4 = nullptr;    // float copy of x for the reduction
    float4* force = nullptr;   // reduction result (F / 48)
    int32_t* ids = nullptr;    // execution slot -> caller's atom id
    int32_t* ids_tmp = nullptr;
    PartitionOut part{};
    irr::Sliced sl{};          // sliced entry layout (when it pays)
    InstDesc* d_inst = nullptr;
    InstDesc inst{};           // host copy of *d_inst (the force launch's parameter)
    WorkItem* d_items = nullptr;
    int num_items = 0;
    int* d_queue = nullptr;
    int* d_status = nullptr;
    double* d_acc = nullptr;   // [4] KE, PE, virial, spare
    int64_t edges = 0;
    int64_t steps = 0;
    int64_t rebuilds = 0;
    int64_t since_rebuild = 0;
    uint32_t row_cap = 0;      // per-node slots for the next rebuild's one-pass search (0: two passes)
    int2* half = nullptr;      // exec_plain: the half list (i < j, execution order) of the rows
};


namespace irr {
// One step of one system, split so a server can batch the force launch:
// md_kick_drift, md_rebuild (when due), the forces (md_forces, or one
// batched launch over md_instance() of many systems), md_kick.
int md_rebuild(irr_md* m);
int md_forces(irr_md* m);
int md_kick_drift(irr_md* m);
int md_kick(irr_md* m);
InstDesc md_instance(const irr_md* m);
// irr_md_destroy, what the pool holds unused left there (a serving loop's next
// system takes it).
void md_free(irr_md* m);
// Digest of the final positions by atom id (a sum of per-atom 64-bit mixes).
int md_state_digest(irr_md* m, uint64_t* digest);
}  // namespace irr
