// Fused RK3 substep of the MHD module: 6th-order stencils of the eight input
// fields, the continuity / momentum / induction / entropy right-hand sides and
// the Williamson 2N update, in one pass.
//
// Reference behaviour being reproduced:
//   kernel body            acc/mhd_solver/stencil_kernel.ac:693-734
//   stencils               acc/stdlib/stdderiv.h:13-262
//   RHS                    acc/mhd_solver/stencil_kernel.ac:355-528
//   2N update, "previous   src/core/kernels/integration.cuh:14-52
//   state" form:  s = 0   : out = in + beta1 * dt * f
//                 s = 1, 2: out = in + beta_{s+1} (alpha_{s+1}/beta_s (in - out) + dt f)
//   forcing (s = 2 only)   acc/mhd_solver/stencil_kernel.ac:611-648,713-717
//                          (STEP 3 = substep 2 with forcing; STEP 2 leaves it out)
//
// B200 structure (no counterpart in the reference, which reads 55 stencil points
// per field straight from global memory with one thread per vertex):
//   - persistent CTAs (one per SM slot) march the columns of x-y tiles
//     round-robin, so the CTAs of one wave stream neighbouring tiles at the same
//     z and read each other's halo planes from L2, and share the planes of the
//     last, partial wave evenly (Pieces; ensembles: a list made by the host);
//   - each CTA streams its tile along z (2.5D): a producer warp issues one TMA
//     load per plane bringing all eight fields of a (TX+8) x (TY+6) halo'd tile
//     into a ring of NP plane slots in shared memory (mbarrier `full` with
//     transaction bytes); consumer warps release a slot through an `empty`
//     mbarrier when done, so no block-wide barrier sits in the plane loop;
//   - single precision: the layout interleaves the fields in pairs with the
//     same stencils, (lnrho, ss), (ux, ax), (uy, ay), (uz, az), so a stencil
//     point of a pair is one 8-byte shared load and its arithmetic runs in
//     packed f32x2 lanes;
//   - one consumer thread per (x, y) column, which keeps register queues along
//     z (values of its column, and running sums of the lower halves of the xz /
//     yz diagonals), so the ring is read for the centre plane and the three
//     above it only (100 8-byte shared loads per vertex in single precision, two
//     fields each, 224 in double precision instead of 296) and a plane's slot
//     is released as soon as its own outputs are done; the centre-only values
//     (previous state, lo parts) arrive by TMA in a ring of output-plane slots
//     (the mixed build) or by plain loads of what was prefetched into L1;
//   - the stencils' coefficients are the same constants on every axis, the
//     leading one (with 1/ds or 1/ds^2) scaling their results; only the 21
//     first, 24 second and 12 cross derivatives the right-hand sides use count;
//   - the mixed build keeps the state as an unevaluated sum hi + lo of a float
//     and a bfloat16 (stored as such, widened to float in registers): stencils
//     read hi, the update is a compensated two-sum.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "tma.cuh"

// What the stencils' results are scaled by and the right-hand sides read: a
// mesh's own in SolveParams, an ensemble member's in the launch's parameters (the
// constant bank in both, where a scalar operation takes them as operands). The
// stencils themselves, their leading coefficients taken out, need no parameter
// (StencilCoefs).
template <typename T>
struct RhsParams {
    T s1[3];                  // first derivative: axis; 3/4 / ds
    T s2[3];                  // second derivative: axis; 3/2 / ds^2, over j_unit
    T perp_u[3], own_u[3];    // s2 times nu (across the component's axis), and times
                              // 4/3 nu + zeta (along it)
    T eta_a[3];               // s2 times eta
    T cond_s[3], cond_l[3];   // s2 times gamma / cp, and times gamma - 1
    T cross_u[3], cross_a[3]; // cross derivative {xy, xz, yz}: 3/8 / (ds ds), times
                              // nu / 3 + zeta, and over j_unit
    T nu, two_nu, zeta;
    // j is formed as mu0 j / j_unit, with j_unit (1 ... 2, make_params) such that s2
    // and cross_a are powers of two, exact, where the spacings are equal. Rounded
    // ones leave all of j off by one factor and the Ohmic heating, its square, by
    // two, which adds up from step to step (mixed 512^3, 53 steps: the entropy
    // 2.0e-7 off instead of 2.8e-7).
    T inv_mu0;  // times j_unit
    T k_ohm;    // eta mu0 / mu0^2, of |mu0 j|^2, times j_unit^2
    T gamma_cp; // gamma / cp
    T inv_cp, gamma, gm1, lnrho0, cs2_sound, k_heat;
    T exp_lnT0; // exp(lnT0): T = exp(lnT0 + E) = exp_lnT0 * exp(E)
#if ACB_MIXED
    T r3[3]; // first derivative's last coefficient: axis (StencilCoefs)
#endif
};

template <typename T>
struct SolveParams {
    RhsParams<T> rhs;
    T rkA, rkB; // out = cur + rkA * (cur - prev) + rkB * rate; rkA unused at s = 0
    // helical forcing, applied after the update at s = 2 when `forcing` != 0
    int forcing;
    T fk[3], ff_re[3], ff_im[3], fcphi, fsphi, fscale, fxs[3], fds[3];
    // time step chosen on the device (acDeviceIntegrateStepCFL): the kernels
    // built with DTDEV take rkB = (T)(rk_beta * *dt_dev) instead of rkB above
    const double* dt_dev;
    double rk_beta;
    // 2 pi / (ds n) per axis in double precision: the single-precision builds
    // form the forcing phase in double (forcing_column, forcing_plane)
    double fxs_d[3];
};

struct SolveGeom {
    Layout L;
    int3 start, end; // region of interior vertices to update, [start, end)
    int tx0;         // index of the first x tile; x tiles are anchored at i = 3 + TX * t
                     // so that every TMA box starts on a 16-byte boundary
    int ntx, nty;    // tiles covering the region
    int nzr;         // planes of the region
    // single mesh: each CTA marches `nfull` whole columns, tiles blockIdx.x +
    // w * gridDim.x; the `rem` tiles left (from tile `rem0`) are cut into
    // `slabs` slabs of `slab_planes` planes, one CTA per tile and slab, and the
    // last `left` planes of each are shared by the other CTAs (see Pieces)
    int nfull, rem0, rem;
    int slabs, slab_planes, left;
    // or (seg_tasks > 0) the columns are cut into segments of zseg planes, dealt
    // round-robin: task t = (segment t / tiles, tile t % tiles)
    int zseg, seg_tasks;
};

// One task of a CTA: planes [z0, z0 + n) of the column of one x-y tile (of one
// member, by its position in the descriptor table, in an ensemble).
struct __align__(16) Piece {
    int tile, z0, n, member;
};

// One member of an ensemble (many independent meshes advanced by one launch):
// the TMA map of its `in` block, its geometry and its buffers.
// Kept in global memory, one table per buffer parity; its parameters travel
// with the launch (EnsSolveArgs::mp).
template <typename T>
struct __align__(128) MemberDesc {
    CUtensorMap tmap;
    SolveGeom g;
    state_t* out;
    lo16_t* in_lo;
    lo16_t* out_lo;
};

template <typename T>
struct SolveArgs {
    SolveGeom g;
    state_t* out;    // out block (previous state at s > 0; result)
    lo16_t* in_lo;   // mixed build: lo block of `in` (bf16, see common.cuh)
    lo16_t* out_lo;  // mixed build: lo block of `out`
    unsigned* status;
    SolveParams<T> P;
    // step diagnostics (kernels built with DIAG): four FP64 partials per CTA,
    // a finishing counter (zero between launches; the last CTA resets it) and
    // the folded result {max |u|^2, min |u|^2, sum |u|^2, sum exp(lnrho)^2}
    double* diag_partials;
    unsigned* diag_counter;
    double* diag_result;
    // ensemble launches only
    const MemberDesc<T>* members;
};

// Members per ensemble launch (a launch's parameters stay within 32 KB; a
// larger ensemble takes one launch per group of members).
constexpr int ACB_ENS_GROUP = 64;

template <typename T>
struct EnsSolveArgs : SolveArgs<T> {
    // the pieces of the group's members that CTA b marches, in order:
    // pieces[first[b]] ... pieces[first[b + 1] - 1]
    const Piece* pieces;
    const int* first;
    RhsParams<T> mp[ACB_ENS_GROUP];      // by position in the group
};

// Centre-only arrays of a substep that the ring does not carry: the previous
// state (s > 0) and, in the mixed build, the lo parts of `in` and (s > 0) of
// `out` (two lo arrays each, bf16). Map slots: 0 = out hi, 1 = in lo, 2 = out lo.
template <int STEP>
struct CentreSet {
    static constexpr bool PREV = STEP > 0;
    static constexpr bool LO   = ACB_MIXED != 0;
    static constexpr int N     = (PREV ? 1 : 0) + (LO ? (PREV ? 2 : 1) : 0);
    // staged by TMA in the single-precision builds' configurations with a
    // centre ring (the mixed build's): the three arrays of substeps 1 and 2
    // and the lo parts of substep 0, whose plain loads left its warps waiting
    // on memory (long-scoreboard stalls 1.66 per issued instruction at 256^3;
    // the 512^3 step 17.43 -> 17.22 ms, same-box A/B)
    static constexpr bool STAGE = N >= 1;
};

struct CentreMaps {
    CUtensorMap m[3]; // (TX, TY, 1, arrays) boxes over out hi, in lo, out lo
};

template <int TX_, int TY_, int NP_, int MINB_, int NC_ = 0>
struct TileCfg {
    static constexpr int TX = TX_, TY = TY_, NP = NP_, MINB = MINB_;
    // NC > 0: the centre-only values of single-mesh single-precision substeps
    // arrive by TMA in a ring of NC output-plane slots (else plain loads)
    static constexpr int NC = NC_;
    static constexpr int CENTRE = TX_ * TY_ * ACB_NARR; // elements of one centre array set
    static constexpr int CENTRE_LO = TX_ * TY_ * ACB_LO_NARR; // the same for a lo block
    static constexpr int BX = TX_ + 8, BY = TY_ + 6;
    static constexpr int CONSUMERS = TX_ * TY_;        // one thread per (x, y) column
    static constexpr int CWARPS    = CONSUMERS / 32;   // consumer warps
    // With 8 or 12 consumer warps the producer is a whole warpgroup (4 warps,
    // one of them working) that hands its registers to the consumers
    // (setmaxnreg), so each consumer thread gets the registers its z queues
    // need. An SM sub-partition's 16K registers hold 2 consumer warps and 1
    // producer warp (2 * 232 + 40 = 504 <= 512 registers a lane), or 3 and 1
    // (3 * 160 + 32 = 512): more warps to hide latency, fewer registers.
    static constexpr bool WGSPEC = CWARPS == 8 || CWARPS == 12;
    static constexpr int THREADS = CONSUMERS + (WGSPEC ? 128 : 32); // plus the producer
    static constexpr int REG_CONSUMER = CWARPS == 12 ? 160 : 232;
    static constexpr int REG_PRODUCER = CWARPS == 12 ? 32 : 40;
    // registers a thread the launch must hold for the reallocation to balance
    static constexpr int REG_LAUNCH =
        WGSPEC ? (REG_CONSUMER * CONSUMERS + REG_PRODUCER * 128 + THREADS - 1) / THREADS : 0;
    static constexpr int FIELD   = BX * BY;           // elements per array of a ring slot
    static constexpr int PLANE   = ACB_NARR * FIELD;  // elements per ring slot
    static constexpr size_t ring_bytes() { return (size_t)NP * PLANE * ACB_ELEM; }
    // prev hi, then (mixed) cur lo and prev lo
    static constexpr size_t centre_slot_bytes()
    {
        return (size_t)(ACB_MIXED ? CENTRE + 2 * CENTRE_LO : CENTRE) * ACB_ELEM;
    }
    static constexpr size_t smem_bytes() { return ring_bytes() + NC * centre_slot_bytes(); }
    // A task starts once the first 2 NGHOST planes are in the ring (the queue
    // priming and the first output plane's upper half): a shallower ring could
    // never hold them.
    static_assert(NP >= 2 * NGHOST, "ring too shallow for the planes a task waits for");
    static_assert(smem_bytes() <= 227 * 1024, "shared memory of one CTA exceeded");
};

namespace acb {

template <typename T>
__device__ __forceinline__ T
rexp(T x)
{
    return exp(x);
}
template <>
__device__ __forceinline__ float
rexp<float>(float x)
{
    return expf(x);
}

// 1 / x: correctly rounded in double precision; in single precision the fast
// division (within 2 ulp of the IEEE quotient for the arguments here, T of order
// one), which avoids the special-case path of the correctly rounded reciprocal
template <typename T>
__device__ __forceinline__ T
rrcp(T x)
{
    return __drcp_rn(x);
}
template <>
__device__ __forceinline__ float
rrcp<float>(float x)
{
    return __fdividef(1.0f, x);
}

// ---- stencil values --------------------------------------------------------
// The stencils are written once over a value type V: a double (one field), or
// F2, the two fields of a pair array in packed FP32 lanes. add/sub/mul/
// fma.rn.f32x2 operate on two independent FP32 lanes with the rounding of the
// scalar operations, so a pair of fields whose stencils have the same shape
// forms its sums and differences in half the instructions; in the layout a pair
// is one array of 8-byte (A, B) elements, so an F2 is also one 8-byte load. The
// rounding sequence is fixed: no operation is left for the compiler to contract,
// so every kernel that uses a function below gets the same bits from it.
struct F2 {
    unsigned long long v;
};

__device__ __forceinline__ F2
pk2(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ void
upk2(F2 r, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r.v));
}

__device__ __forceinline__ F2
add2(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

__device__ __forceinline__ F2
sub2(F2 a, F2 b)
{
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

__device__ __forceinline__ F2
mul2(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

__device__ __forceinline__ F2
fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

__device__ __forceinline__ F2 vadd(F2 a, F2 b) { return add2(a, b); }
__device__ __forceinline__ F2 vsub(F2 a, F2 b) { return sub2(a, b); }
__device__ __forceinline__ F2 vmul(F2 c, F2 b) { return mul2(c, b); }
__device__ __forceinline__ F2 vfma(F2 c, F2 b, F2 d) { return fma2(c, b, d); }
__device__ __forceinline__ double vadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double vsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double vmul(double c, double b) { return __dmul_rn(c, b); }
__device__ __forceinline__ double vfma(double c, double b, double d) { return __fma_rn(c, b, d); }

__device__ __forceinline__ float rfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }

// the value type of a block's arrays
typedef std::conditional<ACB_PAIRED, F2, double>::type V;

// The stencils' coefficients with the leading one taken out, equal on every axis
// (acc/stdlib/stdderiv.h:13-84: 3/4, -3/20, 1/60 of the first derivative; 3/2,
// -3/20, 1/90 and -49/18 of the second; 3/8, -3/80, 1/360 of the cross one):
//   first   d1 + r2 d2 + r3 d3,             r2 = -1/5,  r3 = 1/45
//   second  s1 + q2 s2 + q3 s3 (+ q0 f0),   q2 = -1/10, q3 = 1/135, q0 = -49/27
//   cross   e1 + q2 e2 + q3 e3
// Held in registers for the whole launch: a packed operation takes no constant
// operand, so each of the 45 (c, c) pairs that per-axis coefficients would need
// costs a uniform load and two moves every plane. What depends on the axis scales
// the results, as scalar operations with a constant operand.
//
// Rounded coefficients leave every derivative of a smooth field off by one
// factor, which adds up from step to step where the roundings of the operations
// do not. The mixed build, whose state is fine enough for that to show, takes the
// last coefficient from the sum that the others leave: d_k is about 2 k h f', s_k
// and e_k / 4 about k^2 h^2 f'', so r3 follows from s1 (2 + 4 r2 + 6 r3) = 1 / ds
// with s1 and r2 as rounded, for each axis (RhsParams::r3), and q3 from 1 + 4 q2 +
// 9 q3 = 2/3. They differ from 1/45 and 1/135 by a few units in the last place. At
// 2 pi / 128 first derivatives are then 0.4e-8 off instead of 3.8e-8, and lnrho of
// smooth fields after 53 steps 2.7e-8 instead of 3.6e-8 (2-norm, from FP64); no
// slower (8 steps of 512^3 129.4 against 129.8 ms).
struct StencilCoefs {
    V r2, q0, q2, q3, r3[ACB_MIXED ? 3 : 1];
    template <class PT>
    __device__ __forceinline__ StencilCoefs(const PT& P)
    {
        r2 = value(-1.0 / 5.0);
        q0 = value(-49.0 / 27.0);
        q2 = value(-1.0 / 10.0);
#if ACB_MIXED
        q3 = value((-1.0 / 3.0 - 4.0 * (double)(-1.0f / 10.0f)) / 9.0);
#pragma unroll
        for (int a = 0; a < 3; ++a)
            r3[a] = value(P.r3[a]);
#else
        (void)P;
        q3    = value(1.0 / 135.0);
        r3[0] = value(1.0 / 45.0);
#endif
    }
    __device__ __forceinline__ V third(int axis) const { return r3[ACB_MIXED ? axis : 0]; }
    // opaque, so that it is kept and not formed again at each use
    static __device__ __forceinline__ V
    value(double c)
    {
        V r;
#if AC_DOUBLE_PRECISION == 1
        asm("mov.f64 %0, %1;" : "=d"(r) : "d"(c));
#else
        const float f = (float)c;
        asm volatile("mov.b64 %0, {%1, %1};" : "=l"(r.v) : "f"(f));
#endif
        return r;
    }
};

// d1 + c2 d2 + c3 d3, and the same added to a start value
__device__ __forceinline__ V
sum3(V c2, V c3, const V* d)
{
    return vfma(c3, d[2], vfma(c2, d[1], d[0]));
}

// One array's values at a vertex: centre, and the differences f(+k) - f(-k) and
// sums of the six neighbours of each pencil (axis, k-1).
//
// Second differences of the mixed build as u + v with u = f(+k) - f0, v = f(-k)
// - f0: for a smooth field u and v are exact in FP32 (Sterbenz), so f(+k) + f(-k)
// - 2 f0 keeps its digits instead of cancelling terms of size |c0 f0| (about
// 2.7 f / ds^2); mathematically the same stencil (c0 = -2 (c1 + c2 + c3)). This
// is what brings the mixed build from 2.3e-6 to 2.2e-7 of FP64. It is evaluated as
// S = 2 (f(-k) - f0) + (f(+k) - f(-k)), one fused multiply-add on the two exact
// differences (the first difference is formed anyway). The other builds, whose
// error is that of their state, take the plain sums f(+k) + f(-k) and add c0 f0
// (two operations per point pair instead of three).
// First differences f(+k) - f(-k) directly, as the queues are primed, so
// results do not depend on where a task's z segment starts.
constexpr bool DIFF_FORM = ACB_MIXED != 0;

// Queued values of a column, from plane z+ZQ-4 down to z-3: in double precision
// those below the current plane; in single precision all but the one at z+3, so
// that the 19 values on the axes through a vertex cost 13 shared loads instead of
// 16 (256^3 FP32 substep 0: 477 us, with three queued values 502; substeps 1 and 2
// 520 either way; four to six values in double precision: no gain).
constexpr int ZQ = ACB_PAIRED ? 6 : 3;

template <class V>
struct Pencils {
    V f0, d[3][3], s[3][3];
};

__device__ __forceinline__ void
point_pair(F2 p, F2 m, F2 f0, F2& d, F2& s)
{
    d = sub2(p, m);
    if constexpr (DIFF_FORM)
        s = fma2(F2{0x4000000040000000ull}, sub2(m, f0), d); // (2, 2) * (m - f0) + d
    else
        s = add2(p, m);
}

__device__ __forceinline__ void
point_pair(double p, double m, double, double& d, double& s)
{
    d = __dsub_rn(p, m);
    s = __dadd_rn(p, m);
}

// c: the array's centre element in the centre slot; zo[3..6]: element offsets of
// the slots of planes z .. z+3 from the centre slot; zq: the queued values of the
// thread's own column (ZQ below), to which the value at z+3 is added.
template <class V, int BX>
__device__ __forceinline__ void
load_pencils(const V* __restrict__ c, const int* zo, V* zq, Pencils<V>& p)
{
    // zq[k] is the value at plane z + ZQ - 4 - k
    p.f0 = ZQ > 3 ? zq[ZQ > 3 ? ZQ - 4 : 0] : c[0];
    V zp[3]; // z+1, z+2, z+3
#pragma unroll
    for (int k = 1; k <= 3; ++k)
        zp[k - 1] = k <= ZQ - 4 ? zq[ZQ - 4 - k < 0 ? 0 : ZQ - 4 - k] : c[zo[3 + k]];
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
        point_pair(c[k], c[-k], p.f0, p.d[0][k - 1], p.s[0][k - 1]);
        point_pair(c[k * BX], c[-k * BX], p.f0, p.d[1][k - 1], p.s[1][k - 1]);
    }
#pragma unroll
    for (int k = 1; k <= 3; ++k)
        point_pair(zp[k - 1], zq[ZQ - 4 + k], p.f0, p.d[2][k - 1], p.s[2][k - 1]);
#pragma unroll
    for (int k = ZQ - 1; k > 0; --k)
        zq[k] = zq[k - 1];
    zq[0] = ZQ > 3 ? zp[ZQ > 3 ? ZQ - 4 : 0] : p.f0;
}

// Second derivative along one axis, over its leading coefficient.
__device__ __forceinline__ V
second(const StencilCoefs& K, const Pencils<V>& p, int axis)
{
    const V* s = p.s[axis];
    if constexpr (DIFF_FORM)
        return sum3(K.q2, K.q3, s);
    else
        return vfma(K.q3, s[2], vfma(K.q2, s[1], vfma(K.q0, p.f0, s[0])));
}

// The lower halves of the xz and yz diagonal cross derivatives stream along z.
// The derivative at plane z, over its leading coefficient,
//   sum_k e_k (f(+k,+k) + f(-k,-k) - f(+k,-k) - f(-k,+k))
//     = U(z) - L(z),  U(z) = sum_k e_k d_k(z+k),  L(z) = sum_k e_k d_k(z-k),
// with d_k(w) = f(+k) - f(-k) the x (y) difference at plane w and e = 1, q2, q3:
// the differences of the current plane are formed for the first derivative
// anyway, and each contributes e_k d_k(z) to L(z+k). So a queue keeps
//   a1 = L(z),  a2 = the part of L(z+1) known so far,  a3 = that of L(z+2),
// and advancing a plane is three operations (no register moves):
//   a1 <- a2 + d1(z),  a2 <- a3 + e2 d2(z),  a3 <- e3 d3(z).
// Only the upper half U is read from the ring.
struct LowerSums {
    V a1, a2, a3;
};

// Advances the sums past the plane with differences d.
__device__ __forceinline__ void
push_lower(LowerSums& n, const StencilCoefs& K, const V* d)
{
    n.a1 = vadd(n.a2, d[0]);
    n.a2 = vfma(K.q2, d[1], n.a3);
    n.a3 = vmul(K.q3, d[2]);
}

// The sums at the first plane of a task, from the three planes below it
// (zo[0..2]) of array c's differences along a step (1: x, BX: y), in the order
// in which a streaming task would have added them, so bit for bit the sums it
// would hold.
__device__ __forceinline__ void
prime_lower(LowerSums& n, const StencilCoefs& K, const V* __restrict__ c, const int* zo, int step)
{
    auto d = [&](int plane, int k) { return vsub(c[zo[plane] + k * step], c[zo[plane] - k * step]); };
    n.a1 = vadd(vfma(K.q2, d(1, 2), vmul(K.q3, d(0, 3))), d(2, 1));
    n.a2 = vfma(K.q2, d(2, 2), vmul(K.q3, d(1, 3)));
    n.a3 = vmul(K.q3, d(2, 3));
}

// The z diagonal cross derivative of array c along a step, and its queue advanced
// past the plane (d: the plane's differences along the step).
__device__ __forceinline__ V
z_diagonal(const V* __restrict__ c, const int* zo, int step, const StencilCoefs& K, LowerSums& n,
           const V* d)
{
    V u[3];
#pragma unroll
    for (int k = 1; k <= 3; ++k)
        u[k - 1] = vsub(c[zo[3 + k] + k * step], c[zo[3 + k] - k * step]);
    u[0]      = vsub(u[0], n.a1);
    const V x = sum3(K.q2, K.q3, u);
    push_lower(n, K, d);
    return x;
}

// The derivatives of one array at a vertex, over their leading coefficients:
// gradient, second derivatives by axis, and the cross derivatives that the
// right-hand sides use of a vector's component.
struct Derivs {
    V g[3], d2[3], xa, xb;
};

__device__ __forceinline__ void
gradient_and_second(const StencilCoefs& K, const Pencils<V>& p, Derivs& r)
{
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        r.g[a]  = sum3(K.r2, K.third(a), p.d[a]);
        r.d2[a] = second(K, p, a);
    }
}

// Component I of a vector: a field, or the pair of a velocity and a vector
// potential component. Its cross derivatives with the other axes in order (x
// first); na, nb: the queues of its z diagonals (components 0 and 1: nb; 2: xz in
// na, yz in nb).
template <int I, int BX>
__device__ __forceinline__ void
vector_component(const V* __restrict__ c, const int* zo, V* zq, const StencilCoefs& K,
                 LowerSums& na, LowerSums& nb, V& f0, Derivs& r)
{
    Pencils<V> p;
    load_pencils<V, BX>(c, zo, zq, p);
    f0 = p.f0;
    gradient_and_second(K, p, r);
    if constexpr (I < 2) { // xy diagonals (the whole stencil from the centre plane)
        V e[3];
#pragma unroll
        for (int k = 1; k <= 3; ++k) {
            const int pp = k + k * BX, mm = -k - k * BX, pm = k - k * BX, mp = -k + k * BX;
            e[k - 1] = vsub(vadd(c[pp], c[mm]), vadd(c[pm], c[mp]));
        }
        r.xa = sum3(K.q2, K.q3, e);
        r.xb = z_diagonal(c, zo, I == 0 ? 1 : BX, K, nb, p.d[I]);
    }
    else {
        r.xa = z_diagonal(c, zo, 1, K, na, p.d[0]);
        r.xb = z_diagonal(c, zo, BX, K, nb, p.d[1]);
    }
}

// A scalar (or the pair lnrho, entropy).
template <int BX>
__device__ __forceinline__ void
scalar_field(const V* __restrict__ c, const int* zo, V* zq, const StencilCoefs& K, V& f0, Derivs& r)
{
    Pencils<V> p;
    load_pencils<V, BX>(c, zo, zq, p);
    f0 = p.f0;
    gradient_and_second(K, p, r);
}

// What the right-hand sides are made of (stencil_kernel.ac:355-528, regrouped):
// values and gradients of lnrho and entropy, first = gamma/cp lap s + (gamma-1)
// lap lnrho, velocity and its gradient g[i][a], the off-diagonal sums T of the
// gradient (01, 02, 12), B, mu0 j = grad div A - lap A (over j_unit, RhsParams), the
// viscous terms nu lap u + (nu/3 + zeta) grad div u, eta lap A.
template <typename T>
struct Terms {
    T lnrho, ss, glr[3], gs[3], first;
    T u[3], g[3][3], t01, t02, t12, b[3], j[3];
    T visc[3], resist[3];
};

// Right-hand sides, roc in field order. With E = gamma s/cp + (gamma-1)(lnrho -
// lnrho0), T = exp(lnT0 + E): rho enters only as 1/rho = exp(-lnrho), since the
// heating terms that carry a factor rho are divided by rho T; and both gradients
// in the heat conduction, gamma/cp grad s + (gamma-1) grad lnrho and gamma (grad
// s/cp + grad lnrho) - grad lnrho, are the same vector.
template <typename T, class PT>
__device__ __forceinline__ void
rhs_from(const PT& P, const Terms<T>& m, T roc[ACB_NF])
{
    const T E       = rfma(P.gamma_cp, m.ss, P.gm1 * (m.lnrho - P.lnrho0));
    const T expE    = rexp<T>(E);
    const T cs2     = P.cs2_sound * expE;
    const T inv_rho = rexp<T>(-m.lnrho);
    const T inv_T   = rrcp<T>(P.exp_lnT0 * expE);

    // continuity: -u.grad(lnrho) - div(u). The mixed build sums the products first:
    // added one by one to the divergence, as a rule the larger term, they would
    // round it three times (512^3, 53 steps: lnrho 2.7e-7 off FP64 instead of
    // 2.2e-7). The FP32 build's error is its state's either way, and it is about 1 %
    // faster with one operation less.
    const T divu = m.g[0][0] + m.g[1][1] + m.g[2][2];
    if constexpr (ACB_MIXED)
        roc[0] = -(rfma(m.u[0], m.glr[0], rfma(m.u[1], m.glr[1], m.u[2] * m.glr[2])) + divu);
    else
        roc[0] = -rfma(m.u[0], m.glr[0], rfma(m.u[1], m.glr[1], rfma(m.u[2], m.glr[2], divu)));

    // induction: u x B + eta lap(A)
    roc[4] = rfma(m.u[1], m.b[2], rfma(-m.u[2], m.b[1], m.resist[0]));
    roc[5] = rfma(m.u[2], m.b[0], rfma(-m.u[0], m.b[2], m.resist[1]));
    roc[6] = rfma(m.u[0], m.b[1], rfma(-m.u[1], m.b[0], m.resist[2]));

    // traceless strain: diagonal s, off-diagonal t / 2
    const T third = (T)1 / (T)3;
    const T d3    = third * divu;
    const T s0 = m.g[0][0] - d3, s1 = m.g[1][1] - d3, s2 = m.g[2][2] - d3;

    // momentum: -(u.grad)u - cs2 (grad s / cp + grad lnrho) + j x B / rho +
    //   nu (lap u + grad div u / 3 + 2 S.grad lnrho) + zeta grad div u
    T pr[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
        pr[i] = rfma(P.inv_cp, m.gs[i], m.glr[i]);
    const T jb0 = rfma(m.j[1], m.b[2], -(m.j[2] * m.b[1]));
    const T jb1 = rfma(m.j[2], m.b[0], -(m.j[0] * m.b[2]));
    const T jb2 = rfma(m.j[0], m.b[1], -(m.j[1] * m.b[0]));
    const T sg0 = rfma(s0 + s0, m.glr[0], rfma(m.t01, m.glr[1], m.t02 * m.glr[2]));
    const T sg1 = rfma(m.t01, m.glr[0], rfma(s1 + s1, m.glr[1], m.t12 * m.glr[2]));
    const T sg2 = rfma(m.t02, m.glr[0], rfma(m.t12, m.glr[1], (s2 + s2) * m.glr[2]));
    const T irm = inv_rho * P.inv_mu0;
    auto momentum = [&](int i, T jb, T sg) {
        T r = rfma(-m.u[0], m.g[i][0], m.visc[i]);
        r   = rfma(-m.u[1], m.g[i][1], r);
        r   = rfma(-m.u[2], m.g[i][2], r);
        r   = rfma(P.nu, sg, r);
        r   = rfma(-cs2, pr[i], r);
        return rfma(irm, jb, r);
    };
    roc[1] = momentum(0, jb0, sg0);
    roc[2] = momentum(1, jb1, sg1);
    roc[3] = momentum(2, jb2, sg2);

    // entropy: -u.grad(s) + (eta mu0 j.j + 2 rho nu S:S + zeta rho div(u)^2) / (rho T)
    //   + K / rho (first + |gamma (grad s / cp + grad lnrho) - grad lnrho|^2)
    const T off = rfma(m.t01, m.t01, rfma(m.t02, m.t02, m.t12 * m.t12));
    const T ss  = rfma(s0, s0, rfma(s1, s1, rfma(s2, s2, (T)0.5 * off)));
    const T jj  = rfma(m.j[0], m.j[0], rfma(m.j[1], m.j[1], m.j[2] * m.j[2]));
    const T heat = rfma(P.two_nu, ss, rfma(P.zeta * divu, divu, (P.k_ohm * inv_rho) * jj));
    T cond = m.first;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const T q = rfma(P.gamma, pr[i], -m.glr[i]);
        cond      = rfma(q, q, cond);
    }
    T r    = rfma(inv_T, heat, (P.k_heat * inv_rho) * cond);
    r      = rfma(-m.u[0], m.gs[0], r);
    r      = rfma(-m.u[1], m.gs[1], r);
    roc[7] = rfma(-m.u[2], m.gs[2], r);
}

// Register queues of one thread's column along z: the values of each array at
// the planes of ZQ, and the lower sums of the z diagonals, xz of component 0, yz
// of 1, xz and yz of 2, of (u, A), or of u and then A in double precision.
struct ColumnQ {
    V v[ACB_NARR][ZQ];
    LowerSums n[ACB_PAIRED ? 4 : 8];
};

// Fills the queues from the ring at the first plane of a task (zo[0..2]: the
// three planes below it).
template <int BX, int FIELD>
__device__ __forceinline__ void
prime_queues(const V* __restrict__ c, const int* zo, const StencilCoefs& K, ColumnQ& Q)
{
#pragma unroll
    for (int a = 0; a < ACB_NARR; ++a)
#pragma unroll
        for (int k = 0; k < ZQ; ++k)
            Q.v[a][k] = c[a * FIELD + zo[ZQ - 1 - k]];
#pragma unroll
    for (int w = 0; w < (ACB_PAIRED ? 1 : 2); ++w) {
        const V *x = c + (1 + 3 * w) * FIELD, *y = x + FIELD, *z = y + FIELD;
        prime_lower(Q.n[4 * w + 0], K, x, zo, 1);
        prime_lower(Q.n[4 * w + 1], K, y, zo, BX);
        prime_lower(Q.n[4 * w + 2], K, z, zo, 1);
        prime_lower(Q.n[4 * w + 3], K, z, zo, BX);
    }
}

// Adds the cross derivatives of a vector's components that belong to each
// component of its grad div (k: their coefficients).
template <typename T>
__device__ __forceinline__ void
add_cross_terms(const T* k, const T (&xa)[3], const T (&xb)[3], T (&r)[3])
{
    r[0] = rfma(k[0], xa[1], rfma(k[1], xa[2], r[0]));
    r[1] = rfma(k[0], xa[0], rfma(k[2], xb[2], r[1]));
    r[2] = rfma(k[1], xb[0], rfma(k[2], xb[1], r[2]));
}

// The velocity's terms from its derivatives (g, d2: [component][axis]).
template <typename T>
__device__ __forceinline__ void
velocity_terms(const RhsParams<T>& P, const T (&g)[3][3], const T (&d2)[3][3], const T (&xa)[3],
               const T (&xb)[3], Terms<T>& m)
{
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int a = i == 0 ? 1 : 0, b = i == 2 ? 1 : 2;
#pragma unroll
        for (int x = 0; x < 3; ++x)
            m.g[i][x] = P.s1[x] * g[i][x];
        m.visc[i] = rfma(P.own_u[i], d2[i][i], rfma(P.perp_u[a], d2[i][a], P.perp_u[b] * d2[i][b]));
    }
    add_cross_terms(P.cross_u, xa, xb, m.visc);
    m.t01 = m.g[0][1] + m.g[1][0];
    m.t02 = m.g[0][2] + m.g[2][0];
    m.t12 = m.g[1][2] + m.g[2][1];
}

// The vector potential's: B, eta lap A and mu0 j = grad div A - lap A (over j_unit).
template <typename T>
__device__ __forceinline__ void
potential_terms(const RhsParams<T>& P, const T (&g)[3][3], const T (&d2)[3][3], const T (&xa)[3],
                const T (&xb)[3], Terms<T>& m)
{
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int a = i == 0 ? 1 : 0, b = i == 2 ? 1 : 2;
        m.b[i] = i == 0 ? rfma(P.s1[1], g[2][1], -(P.s1[2] * g[1][2]))
                        : (i == 1 ? rfma(P.s1[2], g[0][2], -(P.s1[0] * g[2][0]))
                                  : rfma(P.s1[0], g[1][0], -(P.s1[1] * g[0][1])));
        m.resist[i] = rfma(P.eta_a[0], d2[i][0], rfma(P.eta_a[1], d2[i][1], P.eta_a[2] * d2[i][2]));
        m.j[i]      = rfma(-P.s2[a], d2[i][a], -(P.s2[b] * d2[i][b]));
    }
    add_cross_terms(P.cross_a, xa, xb, m.j);
}

// Density's and entropy's.
template <typename T>
__device__ __forceinline__ void
scalar_terms(const RhsParams<T>& P, const T (&gl)[3], const T (&gs)[3], const T (&dl)[3],
             const T (&ds)[3], Terms<T>& m)
{
    T f = P.cond_l[0] * dl[0];
    f   = rfma(P.cond_l[1], dl[1], f);
    f   = rfma(P.cond_l[2], dl[2], f);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        f        = rfma(P.cond_s[a], ds[a], f);
        m.glr[a] = P.s1[a] * gl[a];
        m.gs[a]  = P.s1[a] * gs[a];
    }
    m.first = f;
}

// Right-hand sides at one vertex and the centre values of each array; advances
// the queues by a plane. Single precision: the stencils of two fields at once,
// (lnrho, ss), (ux, ax), (uy, ay), (uz, az). `late` is called before the stencils
// of density and entropy, the last.
template <int BX, int FIELD, class F>
__device__ __forceinline__ void
mhd_rhs_q(const V* __restrict__ c, const int* zo, const StencilCoefs& K,
          const RhsParams<AcReal>& P, AcReal roc[ACB_NF], V cur[ACB_NARR], ColumnQ& Q, F late)
{
    typedef AcReal T;
    Terms<T> m;
#if AC_DOUBLE_PRECISION == 0
    T g[2][3][3], d2[2][3][3], xa[2][3], xb[2][3];
    auto component = [&](auto I, LowerSums& na, LowerSums& nb) {
        constexpr int i = I.value;
        Derivs r;
        vector_component<i, BX>(c + (1 + i) * FIELD, zo, Q.v[1 + i], K, na, nb, cur[1 + i], r);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            upk2(r.g[x], g[0][i][x], g[1][i][x]);
            upk2(r.d2[x], d2[0][i][x], d2[1][i][x]);
        }
        upk2(r.xa, xa[0][i], xa[1][i]);
        upk2(r.xb, xb[0][i], xb[1][i]);
        T unused;
        upk2(cur[1 + i], m.u[i], unused);
        (void)unused;
    };
    component(std::integral_constant<int, 0>{}, Q.n[0], Q.n[0]);
    component(std::integral_constant<int, 1>{}, Q.n[1], Q.n[1]);
    component(std::integral_constant<int, 2>{}, Q.n[2], Q.n[3]);
    potential_terms(P, g[1], d2[1], xa[1], xb[1], m);
    velocity_terms(P, g[0], d2[0], xa[0], xb[0], m);
    late();
    Derivs r;
    scalar_field<BX>(c, zo, Q.v[0], K, cur[0], r);
    upk2(cur[0], m.lnrho, m.ss);
    T gl[3], gs[3], dl[3], ds[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        upk2(r.g[x], gl[x], gs[x]);
        upk2(r.d2[x], dl[x], ds[x]);
    }
    scalar_terms(P, gl, gs, dl, ds, m);
#else
    auto vector = [&](int f, LowerSums* n, auto terms) {
        Derivs r[3];
        vector_component<0, BX>(c + f * FIELD, zo, Q.v[f], K, n[0], n[0], cur[f], r[0]);
        vector_component<1, BX>(c + (f + 1) * FIELD, zo, Q.v[f + 1], K, n[1], n[1], cur[f + 1], r[1]);
        vector_component<2, BX>(c + (f + 2) * FIELD, zo, Q.v[f + 2], K, n[2], n[3], cur[f + 2], r[2]);
        T g[3][3], d2[3][3], xa[3], xb[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                g[i][x]  = r[i].g[x];
                d2[i][x] = r[i].d2[x];
            }
            xa[i] = r[i].xa;
            xb[i] = r[i].xb;
        }
        terms(g, d2, xa, xb);
    };
    vector(4, Q.n + 4, [&](auto& g, auto& d2, auto& xa, auto& xb) {
        potential_terms(P, g, d2, xa, xb, m);
    });
    vector(1, Q.n, [&](auto& g, auto& d2, auto& xa, auto& xb) {
        velocity_terms(P, g, d2, xa, xb, m);
    });
    late();
    Derivs l, e;
    scalar_field<BX>(c, zo, Q.v[0], K, cur[0], l);
    scalar_field<BX>(c + 7 * FIELD, zo, Q.v[7], K, cur[7], e);
    m.u[0]  = cur[1];
    m.u[1]  = cur[2];
    m.u[2]  = cur[3];
    m.lnrho = cur[0];
    m.ss    = cur[7];
    scalar_terms(P, l.g, e.g, l.d2, e.d2, m);
#endif
    rhs_from(P, m, roc);
}

// Helical forcing at interior vertex (i, j, k) (stencil_kernel.ac:611-648 with
// a single device: global index = local index, global grid = local grid), the
// double-precision build's; the single-precision builds form the phase by
// parts (forcing_column, forcing_plane and forcing_from below).
template <typename T>
__device__ __forceinline__ void
forcing_at(const SolveParams<T>& P, int i, int j, int k, T f[3])
{
    static_assert(sizeof(T) == 8, "the single-precision builds use forcing_from");
    T skx, ckx;
    const T x0 = (T)(i - NGHOST) * P.fds[0] * P.fxs[0];
    const T x1 = (T)(j - NGHOST) * P.fds[1] * P.fxs[1];
    const T x2 = (T)(k - NGHOST) * P.fds[2] * P.fxs[2];
    const T kx = P.fk[0] * x0 + P.fk[1] * x1 + P.fk[2] * x2;
    sincos(kx, &skx, &ckx);
    const T re = ckx * P.fcphi - skx * P.fsphi;
    const T im = ckx * P.fsphi + skx * P.fcphi;
    bool ok    = true;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        f[c] = P.fscale * (P.ff_re[c] * re - P.ff_im[c] * im);
        ok   = ok && isfinite(f[c]);
    }
    if (!ok)
        f[0] = f[1] = f[2] = 0;
}

// sin and cos of a double-precision phase, reduced to [-pi, pi] in double
// precision first
__device__ __forceinline__ void
sincos_reduced(double ph, float& s, float& c)
{
    const double red = ph - 6.283185307179586 * rint(ph * 0.15915494309189535);
    sincosf((float)red, &s, &c);
}

// The single-precision builds' forcing, by parts: the phase k.x + phi of
// vertex (i, j, k) is (k_x x + k_y y) + k_z z + phi, and exp(i (k.x + phi)) is
// the product of exp(i (k_x x + k_y y + phi)), formed once per column of a task
// (forcing_column), and exp(i k_z z), once per plane (forcing_plane; a warp's
// lanes form 32 planes' at a time, shuffled to the vertex's plane). Each part's
// phase is formed in double precision and reduced before its sin and cos, as
// forcing_at does for the whole phase; the product adds one rounding of a unit
// complex number. The exponentials then cost once per column and plane instead
// of once per vertex (the forced substep 2: 5.79 -> 5.44 ms at 512^3, 49.4 ->
// 46.3 ms at 1024^3, same-box A/B).
template <typename T>
__device__ __forceinline__ void
forcing_column(const SolveParams<T>& P, int i, int j, float& cxy, float& sxy)
{
    const double x0 = ((double)(i - NGHOST) * (double)P.fds[0]) * P.fxs_d[0];
    const double x1 = ((double)(j - NGHOST) * (double)P.fds[1]) * P.fxs_d[1];
    float s, c;
    sincos_reduced((double)P.fk[0] * x0 + (double)P.fk[1] * x1, s, c);
    cxy = c * (float)P.fcphi - s * (float)P.fsphi; // times exp(i phi)
    sxy = s * (float)P.fcphi + c * (float)P.fsphi;
}

template <typename T>
__device__ __forceinline__ void
forcing_plane(const SolveParams<T>& P, int k, float& cz, float& sz)
{
    const double x2 = ((double)(k - NGHOST) * (double)P.fds[2]) * P.fxs_d[2];
    sincos_reduced((double)P.fk[2] * x2, sz, cz);
}

template <typename T>
__device__ __forceinline__ void
forcing_from(const SolveParams<T>& P, float cxy, float sxy, float cz, float sz, T f[3])
{
    const float re = cxy * cz - sxy * sz;
    const float im = sxy * cz + cxy * sz;
    bool ok        = true;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        f[c] = (T)(P.fscale * (P.ff_re[c] * re - P.ff_im[c] * im));
        ok   = ok && isfinite(f[c]);
    }
    if (!ok)
        f[0] = f[1] = f[2] = 0;
}

// Compensated sum of float pairs (hi, lo) and float increments d, two fields
// in packed lanes: a two-sum of hi and d (s and its exact error e), the error
// added to lo, and the result renormalised so that |olo| <= ulp(ohi) / 2.
__device__ __forceinline__ void
pair_add2(F2 hi, F2 lo, F2 d, F2& ohi, F2& olo)
{
    const F2 s  = add2(hi, d);
    const F2 bb = sub2(s, hi);
    const F2 e  = add2(sub2(hi, sub2(s, bb)), sub2(d, bb)); // two-sum error
    const F2 l  = add2(lo, e);
    ohi         = add2(s, l); // renormalise
    olo         = sub2(l, sub2(ohi, s));
}

} // namespace acb

// Step diagnostics of the output state, accumulated per consumer thread while
// the last substep writes it: max, min and sum of |u|^2 and sum of
// exp(lnrho)^2, in FP64 from the stored values (hi + lo in the mixed build),
// each value formed exactly as the reduction kernels form it (reduce.cuh:
// red_load, red_len2, the RMS_EXP filter), so max and min equal a separate
// pass bit for bit (sqrt is monotonic) and the sums differ only in their order.
struct DiagAcc {
    double mx, mn, su, se;
};

__device__ __forceinline__ void
diag_init(DiagAcc& a)
{
    a.mx = -INFINITY;
    a.mn = INFINITY;
    a.su = 0.0;
    a.se = 0.0;
}

__device__ __forceinline__ void
diag_add(DiagAcc& a, double lnrho, double ux, double uy, double uz)
{
    const double l2 = __fma_rn(uz, uz, __fma_rn(uy, uy, __dmul_rn(ux, ux)));
    a.mx            = fmax(a.mx, l2);
    a.mn            = fmin(a.mn, l2);
    a.su += l2;
    const double e = exp(lnrho);
    a.se += e * e;
}

// Values of the vertex's own column that the update needs besides the ring:
// the previous state (s > 0) and, in the mixed build, the lo parts.
// FP64 build: one value per field.
struct CentreVals {
    AcReal prev[ACB_NF];
};

template <int STEP>
__device__ __forceinline__ void
load_centre(const Layout& L, const state_t* out, long long id, CentreVals& c)
{
#pragma unroll
    for (int f = 0; f < ACB_NF; ++f)
        if (STEP > 0)
            c.prev[f] = out[fidx(L, f, id)];
}

// The previous state of the vertex a plane above into L1.
template <int STEP>
__device__ __forceinline__ void
prefetch_centre(const Layout& L, const state_t* out, long long id)
{
#pragma unroll
    for (int f = 0; f < ACB_NF; ++f)
        if (STEP > 0)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(out + fidx(L, f, id)));
}

// The lo parts of pair array ar from a lo element (two bf16x2 words, the
// even array's in the low one) as a float pair, and a float pair as a bf16x2
// word (lane A in the low half); bf16 to float is exact.
__device__ __forceinline__ acb::F2
lo_unpack(unsigned long long e, int ar)
{
    const uint32_t x = (ar & 1) ? (uint32_t)(e >> 32) : (uint32_t)e;
    return acb::pk2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u));
}

__device__ __forceinline__ uint32_t
lo_pack(acb::F2 v)
{
    float a, b;
    acb::upk2(v, a, b);
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a)); // b high, a low
    return r;
}

// Single-precision layout: one (A, B) element per pair array; lo parts in
// the mixed build.
struct CentreVals2 {
    acb::F2 prev[ACB_NARR];
    acb::F2 cur_lo[ACB_NARR];
    acb::F2 prev_lo[ACB_NARR];
};

template <int STEP>
__device__ __forceinline__ void
load_centre2(const Layout& L, const state_t* out, const lo16_t* in_lo, const lo16_t* out_lo,
             long long id, CentreVals2& c)
{
    const acb::F2* o               = reinterpret_cast<const acb::F2*>(out);
    const unsigned long long* il   = reinterpret_cast<const unsigned long long*>(in_lo);
    const unsigned long long* ol   = reinterpret_cast<const unsigned long long*>(out_lo);
#pragma unroll
    for (int a = 0; a < ACB_NARR; ++a) {
        const long long e = a * L.fstride + id;
        if (STEP > 0)
            c.prev[a] = o[e];
#if ACB_MIXED
        const long long el = (a >> 1) * L.fstride + id;
        c.cur_lo[a]        = lo_unpack(il[el], a);
        c.prev_lo[a]       = STEP > 0 ? lo_unpack(ol[el], a) : acb::F2{0ull};
#endif
    }
    (void)il;
    (void)ol;
}

// The same values of the vertex a plane above into L1, while this plane's
// right-hand sides run (their plain loads then hit L1 instead of waiting on
// memory: FP32 512^3 step 13.17 -> 13.07 ms, FP32 ensemble step 5.52 -> 5.41 ms).
template <int STEP>
__device__ __forceinline__ void
prefetch_centre2(const Layout& L, const state_t* out, const lo16_t* in_lo, const lo16_t* out_lo,
                 long long id)
{
    const acb::F2* o             = reinterpret_cast<const acb::F2*>(out);
    const unsigned long long* il = reinterpret_cast<const unsigned long long*>(in_lo);
    const unsigned long long* ol = reinterpret_cast<const unsigned long long*>(out_lo);
#pragma unroll
    for (int a = 0; a < ACB_NARR; ++a) {
        if (STEP > 0)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(o + a * L.fstride + id));
#if ACB_MIXED
        if ((a & 1) == 0) {
            const long long el = (a >> 1) * L.fstride + id;
            asm volatile("prefetch.global.L1 [%0];" ::"l"(il + el));
            if (STEP > 0)
                asm volatile("prefetch.global.L1 [%0];" ::"l"(ol + el));
        }
#endif
    }
    (void)o;
    (void)il;
    (void)ol;
}

// The pieces of a single mesh that this CTA marches, in order: its whole columns,
// dealt round-robin so that the CTAs stream neighbouring tiles at the same z and
// read each other's halos from L2; then its part of the last, partial wave (all
// there is on a mesh of fewer tiles than CTAs), a slab of one column or an even
// share, running from column to column, of the planes below the slabs' end.
struct Pieces {
    int w, p, pend;
    __device__ __forceinline__ Pieces(const SolveGeom& g)
    {
        if (g.seg_tasks > 0) {
            p    = blockIdx.x;
            pend = g.seg_tasks;
            return;
        }
        w                = 0;
        const int nslab  = g.slabs * g.rem; // CTAs with a slab
        const int b      = (int)blockIdx.x - nslab, n = (int)gridDim.x - nslab;
        const long long planes = (long long)g.rem * g.left;
        p    = b < 0 ? 0 : (int)(planes * b / n);
        pend = b < 0 ? 1 : (int)(planes * (b + 1) / n); // a slab: one piece
    }
    __device__ __forceinline__ bool next(const SolveGeom& g, Piece& r)
    {
        if (g.seg_tasks > 0) {
            if (p >= pend)
                return false;
            const int tiles = g.ntx * g.nty, seg = p / tiles;
            r.tile          = p - seg * tiles;
            r.z0            = seg * g.zseg;
            r.n             = min(g.zseg, g.nzr - r.z0);
            p += (int)gridDim.x;
            return true;
        }
        if (w < g.nfull) {
            r.tile = (int)(blockIdx.x + (unsigned)w * gridDim.x);
            r.z0   = 0;
            r.n    = g.nzr;
            ++w;
            return true;
        }
        if (p >= pend)
            return false;
        const int b = (int)blockIdx.x;
        if (b < g.slabs * g.rem) {
            const int s = b / g.rem;
            r.tile      = g.rem0 + (b - s * g.rem);
            r.z0        = s * g.slab_planes;
            r.n         = min(g.slab_planes, g.nzr - r.z0);
            p           = pend;
            return r.n > 0;
        }
        const int col = p / g.left;
        r.tile        = g.rem0 + col;
        r.z0          = g.nzr - g.left + (p - col * g.left);
        r.n           = min(g.nzr - r.z0, pend - p);
        p += r.n;
        return true;
    }
};

// The pieces of this CTA: of a single mesh, or an ensemble's listed ones.
template <bool ENS>
struct PieceList : Pieces {
    __device__ __forceinline__ PieceList(const SolveArgs<AcReal>& a) : Pieces(a.g) {}
    __device__ __forceinline__ bool next(const SolveArgs<AcReal>& a, Piece& r)
    {
        return Pieces::next(a.g, r);
    }
};
template <>
struct PieceList<true> {
    int p, pend;
    __device__ __forceinline__ PieceList(const EnsSolveArgs<AcReal>& a)
    {
        p    = a.first[blockIdx.x];
        pend = a.first[blockIdx.x + 1];
    }
    __device__ __forceinline__ bool next(const EnsSolveArgs<AcReal>& a, Piece& r)
    {
        if (p >= pend)
            return false;
        const int4 v = reinterpret_cast<const int4*>(a.pieces)[p++];
        r.tile       = v.x;
        r.z0         = v.y;
        r.n          = v.z;
        r.member     = v.w;
        return true;
    }
};

template <class Cfg>
struct TaskGeom {
    int i0, j0, k0, nout;
    __device__ __forceinline__ TaskGeom(const SolveGeom& g, const Piece& p)
    {
        const int tile_y = p.tile / g.ntx;
        const int tile_x = p.tile - tile_y * g.ntx;
        i0               = NGHOST + (g.tx0 + tile_x) * Cfg::TX;
        j0               = g.start.y + tile_y * Cfg::TY;
        k0               = g.start.z + p.z0;
        nout             = p.n;
    }
};

__device__ __forceinline__ void
fence_tensormap_acquire(const CUtensorMap* map)
{
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(
                     reinterpret_cast<uint64_t>(map))
                 : "memory");
}

// Stores the periodic images of vertex (i, j, k), whose element in the first array
// is id: the ghost vertices, up to one on each axis and their combinations, that a
// fill of the out block would copy it to (n >= 6 on every axis). For meshes that
// stay in L2, where it replaces the fill of the next substep (launch_solve); in a
// large one the lone 32-byte sectors of the x ghosts cost DRAM more than the fill.
template <class E, int N>
__device__ __forceinline__ void
store_images(const Layout& L, E* __restrict__ out, long long id, int i, int j, int k,
             const E (&r)[N])
{
    const int dx = i < 2 * NGHOST ? L.nx : (i >= L.nx ? -L.nx : 0);
    const int dy = j < 2 * NGHOST ? L.ny : (j >= L.ny ? -L.ny : 0);
    const int dz = k < 2 * NGHOST ? L.nz : (k >= L.nz ? -L.nz : 0);
    auto put = [&](long long d) {
#pragma unroll
        for (int a = 0; a < N; ++a)
            out[a * L.fstride + id + d] = r[a];
    };
    const long long ey = (long long)dy * L.mxp, ez = (long long)dz * L.plane;
    if (dx)
        put(dx);
    if (dy) {
        put(ey);
        if (dx)
            put(ey + dx);
    }
    if (dz) {
        put(ez);
        if (dx)
            put(ez + dx);
        if (dy) {
            put(ez + ey);
            if (dx)
                put(ez + ey + dx);
        }
    }
}

// One task of a consumer warp: the planes of one (tile, z segment) column.
// Waits for the ring, computes and stores every output plane, releases the
// slots, and advances the plane counter q. Returns false if the CTA aborts.
template <class Cfg, int STEP, bool ENS, bool DTDEV, bool DIAG, bool IMAGES, class PT>
__device__ __forceinline__ bool
consume_task(const SolveArgs<AcReal>& a, const SolveGeom& gv, const PT& P,
             const Piece& pc, state_t* out, lo16_t* in_lo, lo16_t* out_lo, const void* ring,
             uint64_t* full, uint64_t* empty, volatile int* abort_flag, uint32_t& q,
             const void* centre, uint64_t* full_c, uint64_t* empty_c, uint32_t& oq,
             DiagAcc& dacc)
{
    using CS          = CentreSet<STEP>;
    constexpr bool CT = Cfg::NC > 0 && !ENS && CS::STAGE;
    using T = AcReal;
    constexpr int TX = Cfg::TX, NP = Cfg::NP, BX = Cfg::BX;
    constexpr int FIELD = Cfg::FIELD, PLANE = Cfg::PLANE;
    const int tid  = threadIdx.x;
    const int lane = tid & 31;
    const int tx   = tid % TX;
    const int ty   = tid / TX;
    const Layout& L = gv.L;
    const TaskGeom<Cfg> tg(gv, pc);
    const int nload = tg.nout + 2 * NGHOST;
    const int i     = tg.i0 + tx;
    const int j     = tg.j0 + ty;
    const bool act  = (i >= gv.start.x) && (i < gv.end.x) && (j < gv.end.y);
    const T rkA     = a.P.rkA;
    T rkB           = a.P.rkB;
    if constexpr (DTDEV) {
        rkB = (T)(a.P.rk_beta * *a.P.dt_dev);
        // formed here, not again at every plane
#if AC_DOUBLE_PRECISION == 1
        asm volatile("" : "+d"(rkB));
#else
        asm volatile("" : "+f"(rkB));
#endif
    }
    // this thread's column in a ring slot (elements)
    const int col = (ty + NGHOST) * BX + (tx + 4);

    bool ok = true;
    for (int l = 0; l < 2 * NGHOST && ok; ++l)
        ok = mbar_wait_bounded(&full[(q + l) % NP], ((q + l) / NP) & 1u);
    ok = __all_sync(0xffffffffu, ok);

    acb::ColumnQ Q;
    const acb::StencilCoefs K(P);
    {
        if (ok && act) {
            const uint32_t sc = (q + NGHOST) % NP;
            int zo[7];
#pragma unroll
            for (int dz = -NGHOST; dz <= NGHOST; ++dz)
                zo[dz + NGHOST] = ((int)((q + NGHOST + dz) % NP) - (int)sc) * PLANE;
            const acb::V* c = reinterpret_cast<const acb::V*>(ring) + (size_t)sc * PLANE + col;
            acb::prime_queues<BX, FIELD>(c, zo, K, Q);
        }
        // the three planes below the first output plane now live in the queues
        __syncwarp();
        if (lane == 0 && ok)
            for (int l = 0; l < NGHOST; ++l)
                mbar_arrive(&empty[(q + l) % NP]);
    }

    // forcing (s = 2 with forcing; single precision): the column's phase factor
    float fcxy = 0.f, fsxy = 0.f, fcz = 0.f, fsz = 0.f;
    if constexpr (STEP == 3 && ACB_PAIRED)
        acb::forcing_column(a.P, i, j, fcxy, fsxy);
    (void)fcxy;
    (void)fsxy;

    for (int p = 0; p < tg.nout; ++p) {
        if (ok) {
            const uint32_t l = q + p + 2 * NGHOST;
            ok = mbar_wait_bounded(&full[l % NP], (l / NP) & 1u);
            ok = __all_sync(0xffffffffu, ok);
        }
        if constexpr (CT) {
            if (ok) {
                ok = mbar_wait_bounded(&full_c[oq % Cfg::NC], (oq / Cfg::NC) & 1u);
                ok = __all_sync(0xffffffffu, ok);
            }
        }
        if (!ok || *abort_flag) {
            if (lane == 0) {
                atomicOr(a.status, (unsigned)ACB_STATUS_TMA_TIMEOUT);
                *abort_flag = 1;
            }
            return false;
        }
        const int k = tg.k0 + p;
        float fcb = 0.f, fsb = 0.f; // the plane's forcing phase factor
        if constexpr (STEP == 3 && ACB_PAIRED) {
            if ((p & 31) == 0) // lane l: plane p + l
                acb::forcing_plane(a.P, k + lane, fcz, fsz);
            fcb = __shfl_sync(0xffffffffu, fcz, p & 31);
            fsb = __shfl_sync(0xffffffffu, fsz, p & 31);
        }
        (void)fcb;
        (void)fsb;
        if (act) {
            const long long id = lidx(L, i, j, k);
            const uint32_t sc  = (q + p + NGHOST) % NP;
            int zo[7];
#pragma unroll
            for (int dz = 0; dz <= NGHOST; ++dz) {
                const int sd    = (int)((q + p + NGHOST + dz) % NP);
                zo[dz + NGHOST] = (sd - (int)sc) * PLANE;
            }
            T fo[3] = {0, 0, 0};
            if constexpr (ACB_PAIRED) {
                // previous state and lo parts of this vertex: plain loads issued
                // first, or after the right-hand sides, which keeps their
                // registers free through the stencils: lo parts, and (CT) what
                // is read from the centre slot
                CentreVals2 cv;
                if constexpr (!CT) {
                    if (!ACB_MIXED)
                        load_centre2<STEP>(L, out, in_lo, out_lo, id, cv);
                    if (p + 1 < tg.nout)
                        prefetch_centre2<STEP>(L, out, in_lo, out_lo, id + L.plane);
                }
                const acb::F2* c = reinterpret_cast<const acb::F2*>(ring) + (size_t)sc * PLANE + col;
                float roc[ACB_NF];
                acb::F2 cur2[ACB_NARR];
                acb::mhd_rhs_q<BX, FIELD>(c, zo, K, P, roc, cur2, Q, [] {});
                if constexpr (!CT && ACB_MIXED)
                    load_centre2<STEP>(L, out, in_lo, out_lo, id, cv);
                if constexpr (STEP == 3)
                    acb::forcing_from<T>(a.P, fcxy, fsxy, fcb, fsb, fo);
                if constexpr (CT) {
                    // from the centre slot the producer filled by TMA
                    // slot: prev hi [array][TY][TX], then cur lo and prev lo
                    // [lo array][TY][TX], 8-byte elements
                    const acb::F2* cs = reinterpret_cast<const acb::F2*>(centre) +
                                        (size_t)(oq % Cfg::NC) * (Cfg::centre_slot_bytes() / 8) +
                                        ty * TX + tx;
                    const unsigned long long* csu =
                        reinterpret_cast<const unsigned long long*>(cs);
                    constexpr int FS  = Cfg::TX * Cfg::TY;
                    constexpr int OCL = CS::PREV ? Cfg::CENTRE : 0; // cur lo
                    constexpr int OPL = OCL + Cfg::CENTRE_LO;       // prev lo
#pragma unroll
                    for (int ar = 0; ar < ACB_NARR; ++ar) {
                        if constexpr (CS::PREV)
                            cv.prev[ar] = cs[ar * FS];
#if ACB_MIXED
                        cv.cur_lo[ar] = lo_unpack(csu[OCL + (ar >> 1) * FS], ar);
                        if constexpr (CS::PREV)
                            cv.prev_lo[ar] = lo_unpack(csu[OPL + (ar >> 1) * FS], ar);
                        else
                            cv.prev_lo[ar] = acb::F2{0ull};
#endif
                    }
                    (void)csu;
                }
                // The update, two fields per instruction (one pair array):
                //   FP32:  out = cur + rkA (cur - prev) + rkB roc  [+ forcing]
                //   mixed: d = rkB roc (+ rkA ((cur - prev) + (cur_lo - prev_lo)))
                //          (hi, lo) = (cur, cur_lo) + d, a two-sum  [+ forcing]
                // Forcing acts on ux, uy, uz, lane 0 of arrays 1-3; the lane of
                // ax, ay, az adds 0 (for the mixed pair, adding 0 to a pair that
                // pair_add2 returned leaves it as it is).
                const acb::F2 rkA2 = acb::pk2(rkA, rkA), rkB2 = acb::pk2(rkB, rkB);
                acb::F2* o2 = reinterpret_cast<acb::F2*>(out);
#if ACB_MIXED
                unsigned long long* ol2 = reinterpret_cast<unsigned long long*>(out_lo);
                uint32_t lo_even = 0; // the even array's bf16x2 word, stored with the odd one's
#endif
                // lane 0 of arrays 0..3 holds lnrho, ux, uy, uz: their stored
                // values for the step diagnostics (hi and, mixed, lo)
                float dh[ACB_NARR], dl[ACB_NARR];
                acb::F2 res[ACB_NARR];
#pragma unroll
                for (int ar = 0; ar < ACB_NARR; ++ar) {
                    const int fa = acb_field(ar, 0), fb = acb_field(ar, 1);
                    const long long e = ar * L.fstride + id;
                    const acb::F2 roc2 = acb::pk2(roc[fa], roc[fb]);
#if ACB_MIXED
                    const acb::F2 l2 = cv.cur_lo[ar];
                    acb::F2 d2       = acb::mul2(rkB2, roc2);
                    if (STEP > 0) {
                        const acb::F2 x = acb::add2(acb::sub2(cur2[ar], cv.prev[ar]),
                                                    acb::sub2(l2, cv.prev_lo[ar]));
                        d2 = acb::fma2(rkA2, x, d2);
                    }
                    acb::F2 h2, w2;
                    acb::pair_add2(cur2[ar], l2, d2, h2, w2);
                    if (STEP == 3 && ar >= 1)
                        acb::pair_add2(h2, w2, acb::pk2(fo[ar - 1], 0.f), h2, w2);
                    o2[e] = h2;
                    res[ar] = h2;
                    const uint32_t wl = lo_pack(w2); // lo rounded to bf16 as stored
                    if (ar & 1)
                        ol2[(ar >> 1) * L.fstride + id] =
                            (unsigned long long)lo_even | ((unsigned long long)wl << 32);
                    else
                        lo_even = wl;
                    if constexpr (DIAG) {
                        float t_;
                        acb::upk2(h2, dh[ar], t_);
                        acb::upk2(lo_unpack(wl, 0), dl[ar], t_);
                    }
#else
                    acb::F2 r;
                    if (STEP == 0)
                        r = acb::fma2(rkB2, roc2, cur2[ar]);
                    else
                        r = acb::fma2(rkB2, roc2,
                                      acb::fma2(rkA2, acb::sub2(cur2[ar], cv.prev[ar]), cur2[ar]));
                    if (STEP == 3 && ar >= 1)
                        r = acb::add2(r, acb::pk2(fo[ar - 1], 0.f));
                    o2[e] = r;
                    res[ar] = r;
                    if constexpr (DIAG) {
                        float t_;
                        acb::upk2(r, dh[ar], t_);
                        dl[ar] = 0.f;
                    }
#endif
                }
                if constexpr (IMAGES)
                    store_images(L, o2, id, i, j, k, res);
                if constexpr (DIAG) {
                    // (double)hi + (double)lo, as the reductions read a value
                    double v[4];
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        v[f] = (double)dh[f];
#if ACB_MIXED
                        v[f] += (double)dl[f];
#endif
                    }
                    diag_add(dacc, v[0], v[1], v[2], v[3]);
                }
                (void)dh;
                (void)res;
                (void)dl;
            }
            else {
                if (p + 1 < tg.nout)
                    prefetch_centre<STEP>(L, out, id + L.plane);
                const state_t* c = reinterpret_cast<const state_t*>(ring) + (size_t)sc * PLANE + col;
                T roc[ACB_NF], cur[ACB_NF];
                // the previous state, prefetched into L1 a plane ago, is loaded
                // before the last two fields' stencils: it arrives under them and
                // holds its registers through the least of the work (256^3
                // substep 1: 1083 us, loaded first 1104, after all 1175)
                CentreVals cv;
                acb::mhd_rhs_q<BX, FIELD>(c, zo, K, P, roc, cur, Q,
                                          [&] { load_centre<STEP>(L, out, id, cv); });
                if constexpr (STEP == 3)
                    acb::forcing_at<T>(a.P, i, j, k, fo);
                T dv[4], res[ACB_NF];
#pragma unroll
                for (int f = 0; f < ACB_NF; ++f) {
                    T r;
                    if (STEP == 0)
                        r = cur[f] + rkB * roc[f];
                    else
                        r = cur[f] + rkA * (cur[f] - cv.prev[f]) + rkB * roc[f];
                    if (STEP == 3 && f >= 1 && f <= 3)
                        r += fo[f - 1];
                    out[fidx(L, f, id)] = r;
                    res[f] = r;
                    if (f < 4)
                        dv[f] = r;
                }
                if constexpr (IMAGES)
                    store_images(L, out, id, i, j, k, res);
                if constexpr (DIAG)
                    diag_add(dacc, (double)dv[0], (double)dv[1], (double)dv[2], (double)dv[3]);
                (void)dv;
                (void)res;
            }
        }
        __syncwarp();
        // the centre plane is done with: what later planes need of it is queued
        if (lane == 0)
            mbar_arrive(&empty[(q + p + NGHOST) % NP]);
        if constexpr (CT) {
            if (lane == 0)
                mbar_arrive(&empty_c[oq % Cfg::NC]);
            ++oq;
        }
    }
    // the planes of the task not released yet
    __syncwarp();
    if (lane == 0)
        for (int l = tg.nout + NGHOST; l < nload; ++l)
            mbar_arrive(&empty[(q + l) % NP]);
    q += nload;
    return true;
}

// Warp-specialised pipeline. Warp CWARPS is the producer: one lane issues one
// TMA load per plane (all 8 fields of the halo'd tile) into a ring of NP
// slots, each guarded by a `full` barrier (transaction bytes) and an `empty`
// barrier on which every consumer warp arrives once it has finished with the
// plane. Consumer warps own one vertex column each and never wait for each
// other except through the ring. Which planes of which tiles a CTA marches:
// Pieces. With ENS every piece names its member, whose map, geometry and buffers
// are read from the descriptor table and whose parameters from the launch.
template <bool ENS>
using SolveKernelArgs = typename std::conditional<ENS, EnsSolveArgs<AcReal>, SolveArgs<AcReal>>::type;

// Folds the consumer threads' step diagnostics: a warp butterfly, the warps
// in order, one partial per CTA, and the last CTA to finish folds the partials
// (its first warp: lane l takes CTAs l, l + 32, ... in order, then a fixed
// butterfly) into a.diag_result. Deterministic; no atomics on data. Every
// consumer warp reaches it, also after an abort (its waits are bounded).
template <class Cfg>
__device__ __forceinline__ void
diag_finish(const SolveArgs<AcReal>& a, DiagAcc d)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        d.mx = fmax(d.mx, __shfl_xor_sync(0xffffffffu, d.mx, o));
        d.mn = fmin(d.mn, __shfl_xor_sync(0xffffffffu, d.mn, o));
        d.su += __shfl_xor_sync(0xffffffffu, d.su, o);
        d.se += __shfl_xor_sync(0xffffffffu, d.se, o);
    }
    __shared__ double wred[Cfg::CWARPS][4];
    __shared__ int dlast;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        wred[warp][0] = d.mx;
        wred[warp][1] = d.mn;
        wred[warp][2] = d.su;
        wred[warp][3] = d.se;
    }
    // the consumer warps only: the producer warps have left
    asm volatile("bar.sync 1, %0;" ::"n"(Cfg::CONSUMERS) : "memory");
    if (threadIdx.x == 0) {
        double r[4] = {wred[0][0], wred[0][1], wred[0][2], wred[0][3]};
        for (int w = 1; w < Cfg::CWARPS; ++w) {
            r[0] = fmax(r[0], wred[w][0]);
            r[1] = fmin(r[1], wred[w][1]);
            r[2] += wred[w][2];
            r[3] += wred[w][3];
        }
        double* p = a.diag_partials + 4 * (size_t)blockIdx.x;
        p[0]      = r[0];
        p[1]      = r[1];
        p[2]      = r[2];
        p[3]      = r[3];
        __threadfence();
        dlast = atomicAdd(a.diag_counter, 1u) == gridDim.x - 1;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(Cfg::CONSUMERS) : "memory");
    if (!dlast || warp != 0)
        return;
    __threadfence();
    const volatile double* v = a.diag_partials;
    double f0 = -INFINITY, f1 = INFINITY, f2 = 0.0, f3 = 0.0;
    for (unsigned b = lane; b < gridDim.x; b += 32) {
        f0 = fmax(f0, v[4 * b + 0]);
        f1 = fmin(f1, v[4 * b + 1]);
        f2 += v[4 * b + 2];
        f3 += v[4 * b + 3];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        f0 = fmax(f0, __shfl_xor_sync(0xffffffffu, f0, o));
        f1 = fmin(f1, __shfl_xor_sync(0xffffffffu, f1, o));
        f2 += __shfl_xor_sync(0xffffffffu, f2, o);
        f3 += __shfl_xor_sync(0xffffffffu, f3, o);
    }
    if (lane == 0) {
        a.diag_result[0] = f0;
        a.diag_result[1] = f1;
        a.diag_result[2] = f2;
        a.diag_result[3] = f3;
        *a.diag_counter  = 0u; // zero for the next launch
        __threadfence();
    }
}

// DTDEV: the time step is read from device memory (SolveParams::dt_dev), for
// steps whose time step the device chooses; single meshes, no forcing.
// IMAGES: the launch also writes the periodic images of its output (single
// meshes, the whole interior, n >= 6 on every axis); its code costs the plane loop
// 3 % even where it is skipped, so the other kernels have none of it.
// DIAG: the launch also folds the step diagnostics of its output (diag_finish);
// single meshes, the last substep over the whole interior.
template <class Cfg, int STEP, bool ENS, bool DTDEV = false, bool DIAG = false,
          bool IMAGES = false>
__global__ void __launch_bounds__(Cfg::THREADS, Cfg::MINB)
    solve_kernel(const __grid_constant__ CUtensorMap tin,
                 const __grid_constant__ SolveKernelArgs<ENS> a,
                 const __grid_constant__ CentreMaps cm)
{
    using T = AcReal;
    constexpr int TX = Cfg::TX, NP = Cfg::NP, BX = Cfg::BX;
    constexpr int FIELD = Cfg::FIELD, PLANE = Cfg::PLANE, CWARPS = Cfg::CWARPS;
    constexpr uint32_t PLANE_BYTES = PLANE * ACB_ELEM;

    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* ring = smem_raw; // NP slots of PLANE_BYTES
    __shared__ __align__(8) uint64_t full[NP];
    __shared__ __align__(8) uint64_t empty[NP];
    // centre ring (CT): one slot per output plane, filled by the producer
    // together with the deepest stencil plane that output needs
    using CS             = CentreSet<STEP>;
    constexpr bool CT    = Cfg::NC > 0 && !ENS && CS::STAGE;
    constexpr int NCS    = CT ? Cfg::NC : 1;
    __shared__ __align__(8) uint64_t full_c[NCS];
    __shared__ __align__(8) uint64_t empty_c[NCS];
    unsigned char* centre = smem_raw + Cfg::ring_bytes(); // NC slots of centre_slot_bytes
    __shared__ volatile int abort_flag;

    const int tid  = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < NP; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], CWARPS);
        }
        for (int s = 0; s < NCS; ++s) {
            mbar_init(&full_c[s], 1);
            mbar_init(&empty_c[s], CWARPS);
        }
        fence_barrier_init();
        abort_flag = 0;
        if (!ENS)
            prefetch_tensormap(&tin);
    }
    __syncthreads();
    grid_wait();

    if constexpr (Cfg::WGSPEC) {
        // whole warpgroups: the first two or three consume, the last produces
        if (warp >= CWARPS)
            asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(Cfg::REG_PRODUCER));
        else
            asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(Cfg::REG_CONSUMER));
    }

    if (warp >= CWARPS) {
        // ------------------------------------------------------------ producer
        if (warp == CWARPS && lane == 0) {
            uint32_t q  = 0;
            uint32_t oq = 0; // output planes whose centre arrays were issued
            bool ok     = true;
            int last_m  = -1;
            PieceList<ENS> pieces(a);
            while (ok) {
                const CUtensorMap* map = &tin;
                const SolveGeom* g     = &a.g;
                Piece pc;
                if (!pieces.next(a, pc))
                    break;
                if constexpr (ENS) {
                    const MemberDesc<T>* md = a.members + pc.member;
                    map                     = &md->tmap;
                    g                       = &md->g;
                    if (pc.member != last_m) {
                        fence_tensormap_acquire(map);
                        prefetch_tensormap(map);
                        last_m = pc.member;
                    }
                }
                const TaskGeom<Cfg> tg(*g, pc);
                const int xt    = g->L.offx + tg.i0 - 4; // a multiple of 16 bytes by construction
                const int yt    = tg.j0 - NGHOST;
                const int nload = tg.nout + 2 * NGHOST;
                for (int l = 0; l < nload; ++l) {
                    const uint32_t s = q % NP, use = q / NP;
                    if (use > 0 && !mbar_wait_bounded(&empty[s], (use - 1) & 1u)) {
                        ok = false;
                        break;
                    }
                    if (abort_flag) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&full[s], PLANE_BYTES);
                    tma_load_4d(ring + (size_t)s * PLANE_BYTES, map, xt, yt, tg.k0 - NGHOST + l, 0,
                                &full[s]);
                    ++q;
                    if constexpr (CT) {
                        // plane l is the top one output l - 6 needs: its centre
                        // arrays go out now, into the next centre slot
                        if (l >= 2 * NGHOST) {
                            const uint32_t sc = oq % Cfg::NC, usec = oq / Cfg::NC;
                            if (usec > 0 && !mbar_wait_bounded(&empty_c[sc], (usec - 1) & 1u)) {
                                ok = false;
                                break;
                            }
                            constexpr uint32_t CB = Cfg::CENTRE * ACB_ELEM;    // prev hi
                            constexpr uint32_t CL = Cfg::CENTRE_LO * ACB_ELEM; // a lo set
                            constexpr uint32_t OC = CS::PREV ? CB : 0;        // cur lo
                            constexpr uint32_t OP = OC + CL;                   // prev lo
                            constexpr uint32_t TXB = (CS::PREV ? CB : 0) + (CS::LO ? CL : 0) +
                                                     ((CS::LO && CS::PREV) ? CL : 0);
                            unsigned char* dst = centre + (size_t)sc * Cfg::centre_slot_bytes();
                            const int xc = g->L.offx + tg.i0; // interior tile start: 32-byte aligned
                            const int zc = tg.k0 + (l - 2 * NGHOST);
                            mbar_arrive_expect_tx(&full_c[sc], TXB);
                            if (CS::PREV)
                                tma_load_4d(dst, &cm.m[0], xc, tg.j0, zc, 0, &full_c[sc]);
                            if (CS::LO)
                                tma_load_4d(dst + OC, &cm.m[1], xc, tg.j0, zc, 0, &full_c[sc]);
                            if (CS::LO && CS::PREV)
                                tma_load_4d(dst + OP, &cm.m[2], xc, tg.j0, zc, 0, &full_c[sc]);
                            ++oq;
                        }
                    }
                }
            }
            if (!ok) {
                atomicOr(a.status, (unsigned)ACB_STATUS_TMA_TIMEOUT);
                abort_flag = 1;
                // wait (bounded) for this CTA's loads still in flight before leaving
                for (uint32_t r = q > (uint32_t)NP ? q - NP : 0; r < q; ++r)
                    (void)mbar_wait_bounded(&full[r % NP], (r / NP) & 1u);
                if constexpr (CT)
                    for (uint32_t r = oq > (uint32_t)Cfg::NC ? oq - Cfg::NC : 0; r < oq; ++r)
                        (void)mbar_wait_bounded(&full_c[r % Cfg::NC], (r / Cfg::NC) & 1u);
            }
        }
        return;
    }

    // ---------------------------------------------------------------- consumers
    uint32_t q = 0, oq = 0;
    DiagAcc dacc;
    diag_init(dacc);
    PieceList<ENS> pieces(a);
    Piece pc;
    while (pieces.next(a, pc)) {
        bool ok;
        if constexpr (ENS) {
            // the member's descriptor, and its parameters from the launch
            const MemberDesc<T>* md = a.members + pc.member;
            const SolveGeom gv      = md->g;
            ok = consume_task<Cfg, STEP, ENS, DTDEV, false, false>(a, gv, a.mp[pc.member], pc, md->out,
                                                            md->in_lo, md->out_lo, ring, full,
                                                            empty, &abort_flag, q, centre, full_c,
                                                            empty_c, oq, dacc);
        }
        else {
            ok = consume_task<Cfg, STEP, ENS, DTDEV, DIAG, IMAGES>(a, a.g, a.P.rhs, pc, a.out, a.in_lo, a.out_lo,
                                                    ring, full, empty, &abort_flag, q, centre,
                                                    full_c, empty_c, oq, dacc);
        }
        if (!ok) {
            if constexpr (DIAG)
                break; // every consumer warp still reaches the fold
            else
                return;
        }
    }
    if constexpr (DIAG)
        diag_finish<Cfg>(a, dacc);
}
