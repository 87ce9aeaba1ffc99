// Single-pass reductions over the interior: MAX, MIN, RMS (raw sum of
// squares), RMS_EXP (raw sum of exp^2), SUM, for one field, a vector of three
// fields (by length), or the Alfven speed of three fields plus a density.
//
// Reference behaviour (src/core/kernels/reductions.cuh:18-343, device layer
// src/core/device.cc:477-537): filter functions
//     scalar  v, v^2, exp(v)^2
//     vector  |v|, |v|^2, sum_i exp(v_i)^2         (SUM of a vector sums |v|)
//     Alfven  |B| / sqrt(4 pi exp(rho)),  |B|^2 / (4 pi exp(rho))
// over [n_min, n_max); the device layer returns the unnormalised sum for RMS
// and RMS_EXP.
//
// The reference runs a filter kernel into an n^3 scratch array, a 128-wide
// shared-memory tree, then a single thread folding n^3/128 partials serially,
// all accumulating in AcReal. Here: one kernel, one read of each input; per
// thread FP64 accumulation over warp-owned rows, a warp-shuffle tree, a block
// tree, one FP64 partial per block in scratch, and the last block to finish
// folds the partials in a fixed order (deterministic, no atomics on data).
#pragma once
#include "common.cuh"
#include "tma.cuh"

enum { RED_SCAL = 1, RED_VEC = 3, RED_ALFVEN = 4 };

// sets of one multi-set pass at most: a vector and six scalar fields
constexpr int ACB_RED_SETS = 7;
// entries a Device keeps of the passes on its current block (all eight fields
// and a vector, with room to spare)
constexpr int ACB_RED_RECORD = 16;

// Parameters of the Courant time step, and its record: dt of the last step,
// simulated time, steps taken.
struct CflParams {
    double cdt, cdtv, dsmin, cs2, nu, eta, gamma;
    AcReal timescale;
};

__device__ __forceinline__ void
cfl_step(double umax, const CflParams& p, double* rec)
{
    const double u       = (double)(AcReal)umax;
    const double uu_dt   = p.cdt * p.dsmin / (fabs(u) + sqrt(p.cs2));
    const double visc_dt = p.cdtv * p.dsmin * p.dsmin / fmax(fmax(p.nu, p.eta), fmax(p.gamma, 0.0));
    const AcReal dt      = p.timescale * (AcReal)fmin(uu_dt, visc_dt);
    rec[0]               = (double)dt;
    rec[1] += (double)dt;
    rec[2] += 1.0;
}

struct ReduceArgs {
    Layout L;
    const state_t* f[6];
    const lo16_t* lo[6]; // mixed build: lo parts, lo_field views (else null)
    int nin;            // 1, 3 or 4
    int rtype;          // ReductionType
    int3 start, end;
    long long rows;
    double* partials;   // gridDim.x doubles of scratch
    unsigned* counter;  // scratch counter, zero between launches
    double* result;
    double* cfl_rec; // not null: the last block also takes the time step that
    CflParams cfl;   // set 0's maximum (max |u|) allows
};

__device__ __forceinline__ double
red_combine(int rtype, double a, double b)
{
    if (rtype == RTYPE_MAX || rtype == RTYPE_ALFVEN_MAX)
        return fmax(a, b);
    if (rtype == RTYPE_MIN || rtype == RTYPE_ALFVEN_MIN)
        return fmin(a, b);
    return a + b;
}

__device__ __forceinline__ double
red_identity(int rtype)
{
    if (rtype == RTYPE_MAX || rtype == RTYPE_ALFVEN_MAX)
        return -INFINITY;
    if (rtype == RTYPE_MIN || rtype == RTYPE_ALFVEN_MIN)
        return INFINITY;
    return 0.0;
}

__device__ __forceinline__ double
red_load(const ReduceArgs& a, int w, long long id)
{
    // a.f[w] is the field's base in the block: its vertex id is ACB_LANES
    // values further per element
    double v = (double)a.f[w][id * ACB_LANES];
#if ACB_MIXED
    v += (double)lo16_to_float(a.lo[w][id * ACB_LO_STEP]);
#endif
    return v;
}

// Both fields of the pair array of input w, one 8-byte element: input w's own
// value and its partner's.
__device__ __forceinline__ void
red_load_pair(const ReduceArgs& a, int w, long long id, double& own, double& other)
{
#if AC_DOUBLE_PRECISION == 0
    // the field's base is its array's, or one value further (lane 1)
    const unsigned lane  = (unsigned)(((uintptr_t)a.f[w] >> 2) & 1u);
    const float2 e       = reinterpret_cast<const float2*>(a.f[w] - lane)[id];
    own                  = (double)(lane ? e.y : e.x);
    other                = (double)(lane ? e.x : e.y);
#if ACB_MIXED
    // likewise the pair's bf16x2 word of the lo element
    const uint32_t l = *reinterpret_cast<const uint32_t*>(a.lo[w] - lane + id * ACB_LO_STEP);
    const uint32_t x = l << 16, y = l & 0xffff0000u;
    own += (double)__uint_as_float(lane ? y : x);
    other += (double)__uint_as_float(lane ? x : y);
#endif
#else
    own = other = red_load(a, w, id);
#endif
}

// |v|^2 of a vector, with one fixed rounding sequence for every reduction
// that uses it (the length for MAX / MIN, the square for RMS), so that a pass
// computing several of them returns what separate passes return, bit for bit.
__device__ __forceinline__ double
red_len2(double x, double y, double z)
{
    return __fma_rn(z, z, __fma_rn(y, y, __dmul_rn(x, x)));
}

// The filtered value of one vertex from its nin input values.
template <int NIN>
__device__ __forceinline__ double
red_filter(int rt, const double* v)
{
    if (NIN == RED_SCAL) {
        if (rt == RTYPE_RMS)
            return __dmul_rn(v[0], v[0]);
        if (rt == RTYPE_RMS_EXP) {
            const double e = exp(v[0]);
            return e * e;
        }
        return v[0]; // MAX, MIN, SUM
    }
    const double x = v[0], y = v[1], z = v[2];
    if (NIN == RED_VEC) {
        if (rt == RTYPE_RMS)
            return red_len2(x, y, z);
        if (rt == RTYPE_RMS_EXP) {
            const double ex = exp(x), ey = exp(y), ez = exp(z);
            return ex * ex + ey * ey + ez * ez;
        }
        return sqrt(red_len2(x, y, z)); // MAX, MIN, SUM of the length
    }
    // Alfven speed with density exponent d
    const double d  = v[3];
    const double b2 = x * x + y * y + z * z;
    const double q  = 4.0 * M_PI * exp(d);
    if (rt == RTYPE_ALFVEN_RMS)
        return b2 / q;
    return sqrt(b2) / sqrt(q);
}

// Calls f(values) for every vertex of the rows of this warp, a lane's vertices
// in ascending order. A lane loads its next ACB_RED_AHEAD vertices' inputs
// before it uses the first, so that a row is a few waits on memory instead of one
// for each 32 vertices. 512^3, against one vertex at a time: |u| alone FP32 504 us
// instead of 682, mixed 836 instead of 882, FP64 598 instead of 671; the vector with
// all fields it reads 874, 1068 and 572 us instead of 1340, 1646 and 960; rms_exp
// 324, 337 and 269 instead of 386, 915 and 506; a field with its partner takes 7 to
// 14 % longer, 285 us in FP32.
constexpr int ACB_RED_AHEAD = 4;

template <int THREADS, int NF, class Load, class F>
__device__ __forceinline__ void
red_rows(const ReduceArgs& a, Load load, F f)
{
    const int lane    = threadIdx.x & 31;
    const unsigned gw = (blockIdx.x * THREADS + threadIdx.x) >> 5;
    const unsigned nw = (gridDim.x * THREADS) >> 5;
    const int rx      = a.end.x - a.start.x;
    const unsigned ry = (unsigned)(a.end.y - a.start.y);
    for (unsigned r = gw; r < (unsigned)a.rows; r += nw) {
        const unsigned kq    = r / ry;
        const long long base = lidx(a.L, a.start.x, a.start.y + (int)(r - kq * ry),
                                    a.start.z + (int)kq);
        int i = lane;
        for (; i + 32 * (ACB_RED_AHEAD - 1) < rx; i += 32 * ACB_RED_AHEAD) {
            double v[ACB_RED_AHEAD][NF];
#pragma unroll
            for (int u = 0; u < ACB_RED_AHEAD; ++u)
                load(base + i + 32 * u, v[u]);
#pragma unroll
            for (int u = 0; u < ACB_RED_AHEAD; ++u)
                f(v[u]);
        }
        for (; i < rx; i += 32) {
            double v[NF];
            load(base + i, v);
            f(v);
        }
    }
}

template <int THREADS, int NIN>
__global__ void __launch_bounds__(THREADS)
reduce_kernel(const ReduceArgs a)
{
    const int lane = threadIdx.x & 31;
    const int wid  = threadIdx.x >> 5;
    double acc     = red_identity(a.rtype);
    red_rows<THREADS, NIN>(
        a,
        [&](long long id, double* v) {
#pragma unroll
            for (int w = 0; w < NIN; ++w)
                v[w] = red_load(a, w, id);
        },
        [&](const double* v) { acc = red_combine(a.rtype, acc, red_filter<NIN>(a.rtype, v)); });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        acc = red_combine(a.rtype, acc, __shfl_xor_sync(0xffffffffu, acc, o));
    __shared__ double wsum[THREADS / 32];
    __shared__ bool last;
    if (lane == 0)
        wsum[wid] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = wsum[0];
        for (int w = 1; w < THREADS / 32; ++w)
            b = red_combine(a.rtype, b, wsum[w]);
        a.partials[blockIdx.x] = b;
        __threadfence();
        const unsigned done = atomicAdd(a.counter, 1u);
        last                = (done == gridDim.x - 1);
    }
    __syncthreads();
    if (last) {
        // fixed-order fold of the partials: lanes stride, then a fixed tree
        __threadfence();
        double v = red_identity(a.rtype);
        for (int b = threadIdx.x; b < (int)gridDim.x; b += THREADS)
            v = red_combine(a.rtype, v, ((volatile double*)a.partials)[b]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            v = red_combine(a.rtype, v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0)
            wsum[wid] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            double b = wsum[0];
            for (int w = 1; w < THREADS / 32; ++w)
                b = red_combine(a.rtype, b, wsum[w]);
            *a.result  = b;
            *a.counter = 0u; // ready for the next launch on this stream
        }
    }
}

// MAX, MIN and the RMS sum of one or several sets in one pass: set 0 is one
// scalar field (NIN = RED_SCAL, input 0) or one vector's length (NIN = RED_VEC,
// inputs 0-2); sets 1 .. NS-1 are the scalar fields of the inputs that follow
// (input s for a scalar request, s - 1 for a vector one): the vector's
// components and, in the single-precision builds, the fields that share their
// 8-byte elements (input NIN + w that of input w), whose bytes the pass reads
// anyway. Every set's accumulators are combined in the order in which
// reduce_kernel combines its one, so each equals a pass of its own, bit for bit;
// a vector's MAX and MIN are kept as |v|^2 until the end (sqrt is monotonic and
// correctly rounded, so the root of the largest square is the largest length).
// partials holds 3 * NS * gridDim.x doubles, result 3 * NS (set s at 3 s).
template <int THREADS, int NIN, int NS>
__global__ void __launch_bounds__(THREADS)
reduce_sets_kernel(const ReduceArgs a)
{
    constexpr int NF = NIN == RED_SCAL ? NS : (NS - 1 > 3 ? NS - 1 : 3); // inputs
    static_assert(NF <= 6, "at most six inputs");
    const int lane = threadIdx.x & 31;
    const int wid  = threadIdx.x >> 5;
    double mx[NS], mn[NS], sm[NS];
#pragma unroll
    for (int t = 0; t < NS; ++t) {
        mx[t] = -INFINITY;
        mn[t] = INFINITY;
        sm[t] = 0.0;
    }
    grid_wait();
    red_rows<THREADS, NF>(
        a,
        [&](long long id, double* v) {
            if (ACB_PAIRED && NF == 2 * NIN)
#pragma unroll
                for (int w = 0; w < NIN; ++w)
                    red_load_pair(a, w, id, v[w], v[NIN + w]);
            else
#pragma unroll
                for (int w = 0; w < NF; ++w)
                    v[w] = red_load(a, w, id);
        },
        [&](const double* v) {
#pragma unroll
            for (int t = 0; t < NS; ++t) {
                double m, q;
                if (t == 0 && NIN == RED_VEC)
                    m = q = red_len2(v[0], v[1], v[2]);
                else {
                    m = v[NIN == RED_SCAL ? t : t - 1];
                    q = __dmul_rn(m, m);
                }
                mx[t] = fmax(mx[t], m);
                mn[t] = fmin(mn[t], m);
                sm[t] = sm[t] + q;
            }
        });
#pragma unroll
    for (int t = 0; t < NS; ++t)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mx[t] = fmax(mx[t], __shfl_xor_sync(0xffffffffu, mx[t], o));
            mn[t] = fmin(mn[t], __shfl_xor_sync(0xffffffffu, mn[t], o));
            sm[t] = sm[t] + __shfl_xor_sync(0xffffffffu, sm[t], o);
        }
    __shared__ double wmx[NS][THREADS / 32], wmn[NS][THREADS / 32], wsm[NS][THREADS / 32];
    __shared__ bool last;
    if (lane == 0)
#pragma unroll
        for (int t = 0; t < NS; ++t) {
            wmx[t][wid] = mx[t];
            wmn[t][wid] = mn[t];
            wsm[t][wid] = sm[t];
        }
    __syncthreads();
    const unsigned G = gridDim.x;
    if (threadIdx.x == 0) {
        for (int t = 0; t < NS; ++t) {
            double bx = wmx[t][0], bn = wmn[t][0], bs = wsm[t][0];
            for (int w = 1; w < THREADS / 32; ++w) {
                bx = fmax(bx, wmx[t][w]);
                bn = fmin(bn, wmn[t][w]);
                bs = bs + wsm[t][w];
            }
            a.partials[(3 * t) * G + blockIdx.x]     = bx;
            a.partials[(3 * t + 1) * G + blockIdx.x] = bn;
            a.partials[(3 * t + 2) * G + blockIdx.x] = bs;
        }
        __threadfence();
        const unsigned done = atomicAdd(a.counter, 1u);
        last                = (done == G - 1);
    }
    __syncthreads();
    if (last) {
        // the fixed-order fold of reduce_kernel, for each accumulator
        __threadfence();
        const volatile double* P = a.partials;
        for (int t = 0; t < NS; ++t) {
            double vx = -INFINITY, vn = INFINITY, vs = 0.0;
            for (int b = threadIdx.x; b < (int)G; b += THREADS) {
                vx = fmax(vx, P[(3 * t) * G + b]);
                vn = fmin(vn, P[(3 * t + 1) * G + b]);
                vs = vs + P[(3 * t + 2) * G + b];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                vx = fmax(vx, __shfl_xor_sync(0xffffffffu, vx, o));
                vn = fmin(vn, __shfl_xor_sync(0xffffffffu, vn, o));
                vs = vs + __shfl_xor_sync(0xffffffffu, vs, o);
            }
            if (lane == 0) {
                wmx[t][wid] = vx;
                wmn[t][wid] = vn;
                wsm[t][wid] = vs;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int t = 0; t < NS; ++t) {
                double bx = wmx[t][0], bn = wmn[t][0], bs = wsm[t][0];
                for (int w = 1; w < THREADS / 32; ++w) {
                    bx = fmax(bx, wmx[t][w]);
                    bn = fmin(bn, wmn[t][w]);
                    bs = bs + wsm[t][w];
                }
                if (t == 0 && NIN == RED_VEC) { // (an identity stays one)
                    bx = bx < 0.0 ? bx : sqrt(bx);
                    bn = sqrt(bn);
                }
                a.result[3 * t]     = bx;
                a.result[3 * t + 1] = bn;
                a.result[3 * t + 2] = bs;
                if (t == 0 && a.cfl_rec)
                    cfl_step(bx, a.cfl, a.cfl_rec);
            }
            *a.counter = 0u; // ready for the next launch on this stream
        }
    }
}
