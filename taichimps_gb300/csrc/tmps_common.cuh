// Shared device helpers for the GB300 DEM contact path (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/taichimps_gb300.h"

#define TMPS_DEV __device__ __forceinline__

// Bits 27..31 of a neighbor entry carry the stencil offset of the partner's
// cell relative to the row atom's cell, (ox+1) + 3 (oy+1) + 9 (oz+1); the low
// 27 bits are the partner's internal index (n < 2^27 atoms).
constexpr int kNbrIndexBits = 27;
constexpr int32_t kNbrIndexMask = (1 << kNbrIndexBits) - 1;
constexpr int kMaxSlots = 64;  // one bit per slot in the touch mask

namespace tmps {

// Number of kernels this library has launched (all entry points, all
// threads); read through tmps_launch_count().
void note_launches(int k);

// start[0..m] = exclusive scan of count[0..m), start[m] the total; tile_sum:
// one word per 4,096 of them (two launches, tmps_nlist.cu).
void exclusive_scan(const int32_t* count, int32_t* start, int32_t* tile_sum, int m, cudaStream_t s);

inline int sm_count() {
    static const int sms = [] {
        int dev = 0, v = 0;
        return cudaGetDevice(&dev) == cudaSuccess &&
                       cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0
                   ? v
                   : 152;
    }();
    return sms;
}
// One wave of resident blocks: the occupancy of a kernel times the SMs.
template <typename K>
int wave_blocks(K kernel, int block) {
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, block, 0) != cudaSuccess || occ < 1) occ = 1;
    return occ * sm_count();
}

inline int grid_for(int64_t n, int block) {
    int64_t g = (n + block - 1) / block;
    return (int)(g < 1 ? 1 : g);
}

// A double as an FP32 value from its bits alone: the sign, the exponent
// rebiased and the top 20 bits of the significand (the rest truncated), so
// the relative error is below 2^-20; zero below the FP32 normal range,
// infinity above it, NaN kept.  Integer operations only: on this part a
// double -> float conversion issues on the narrow FP64 pipe, and screens that
// reject far pairs before an exact FP64 test do not need a rounded value.
TMPS_DEV float approx_f32(double x) {
    const uint32_t hi = (uint32_t)__double2hiint(x);
    const uint32_t sign = hi & 0x80000000u;
    const int e = (int)((hi >> 20) & 0x7ffu);
    const uint32_t m = hi & 0xfffffu;
    if (e == 0x7ff) return __uint_as_float(sign | 0x7f800000u | (m ? 0x400000u : 0u));
    const int ef = e - 1023 + 127;
    if (ef <= 0) return __uint_as_float(sign);
    if (ef >= 255) return __uint_as_float(sign | 0x7f800000u);
    return __uint_as_float(sign | ((uint32_t)ef << 23) | (m << 3));
}

// |a| + |b| + |c|
TMPS_DEV float l1f(float a, float b, float c) { return (fabsf(a) + fabsf(b)) + fabsf(c); }

// Conversions between double and float done with integer operations, which
// issue on the wide integer pipes instead of this part's narrow FP64 pipe.
// Both give the same bits as the hardware conversion; the rare operands
// outside the plain case (results below the FP32 normal range, infinities,
// NaNs) go to the hardware conversion.

// isfinite(x) from the exponent bits
TMPS_DEV bool finite_bits(double x) { return ((__double2hiint(x) >> 20) & 0x7ff) != 0x7ff; }

// (float)x, round to nearest even
TMPS_DEV float f32_rn(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const uint32_t sign = (uint32_t)(b >> 32) & 0x80000000u;
    if ((b << 1) == 0ull) return __uint_as_float(sign);  // +-0
    const int e = (int)((b >> 52) & 0x7ff);
    const int ef = e - 1023 + 127;
    if (e == 0x7ff || ef <= 0 || ef >= 255) return (float)x;
    const unsigned long long m = b & 0xfffffffffffffull;
    uint32_t keep = (uint32_t)(m >> 29);
    const uint32_t rest = (uint32_t)(m & 0x1fffffffull);
    if (rest > 0x10000000u || (rest == 0x10000000u && (keep & 1u))) ++keep;
    // a carry out of the significand steps the exponent (to infinity past the top)
    return __uint_as_float(sign | (((uint32_t)ef << 23) + keep));
}

// (double)f, exact
TMPS_DEV double f64_of(float f) {
    const uint32_t u = __float_as_uint(f);
    const unsigned long long sign = (unsigned long long)(u & 0x80000000u) << 32;
    const uint32_t e = (u >> 23) & 0xffu;
    if (e == 0u || e == 0xffu) {
        if ((u << 1) == 0u) return __longlong_as_double((long long)sign);  // +-0
        return (double)f;
    }
    const unsigned long long m = (unsigned long long)(u & 0x7fffffu) << 29;
    return __longlong_as_double((long long)(sign | ((unsigned long long)(e - 127 + 1023) << 52) | m));
}

// hi + lo of a double as two floats: hi = (float)v, lo = (float)(v - hi)
// (v - hi is exact in FP64)
TMPS_DEV void split_dw(double v, float& hi, float& lo) {
    hi = f32_rn(v);
    lo = f32_rn(__dsub_rn(v, f64_of(hi)));
}

// FP64 quotients, reciprocals and square roots, rounded as the operations
// themselves.  This part issues an FP64 instruction for a warp every 16 cycles
// per SM, and the compiler's division and square root are some ten to twenty
// of them each.  These start from the hardware's 20-bit approximations
// (rcp.approx, rsqrt.approx: not on the FP64 pipe) and take one third-order
// step -- Halley's iteration, whose error is the cube of the seed's -- and one
// correction by the exact residual (Markstein 1990): six FP64 instructions a
// quotient (three for each further one by the same divisor), five a
// reciprocal, nine a root.  Before its last rounding a result is within 2^-48
// units in the last place of the exact one, so it is the correctly rounded one
// unless the exact one lies that close to the middle of two neighbours.
// Arguments outside 2^+-1000 (quotients: 2^+-500), zeros, infinities and NaNs
// take the operation itself.
TMPS_DEV bool plain64(double x) {
    const int e = (__double2hiint(x) >> 20) & 0x7ff;
    return e >= 23 && e <= 2023;
}

// 1 / x within 0.51 units in the last place (x plain)
TMPS_DEV double near_rcp64(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = __fma_rn(-x, y, 1.0);
    return __fma_rn(y, __fma_rn(e, e, e), y);
}
// 1 / x from y, a few units in the last place off (x plain)
TMPS_DEV double refine_rcp64(double x, double y) { return __fma_rn(__fma_rn(-x, y, 1.0), y, y); }

// 1 / x
TMPS_DEV double rcp64(double x) {
    if (!plain64(x)) return 1.0 / x;
    return refine_rcp64(x, near_rcp64(x));
}

// a / b with y = 1 / b within two units in the last place at hand: the product
// corrected by its residual, at three dependent FP64 instructions instead of a
// division's latency.  Operands outside 2^+-500 take the division.
TMPS_DEV double div_by(double a, double b, double y) {
    const int ha = __double2hiint(a), ea = (ha >> 20) & 0x7ff, eb = (__double2hiint(b) >> 20) & 0x7ff;
    const bool zero = ((ha & 0x7fffffff) | __double2loint(a)) == 0;
    if (((ea < 523 || ea > 1523) && !zero) || eb < 523 || eb > 1523) return a / b;
    const double q = __dmul_rn(a, y);
    if (zero) return q;  // with its sign, as the quotient's
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}
// a / b
TMPS_DEV double quot64(double a, double b) { return div_by(a, b, near_rcp64(b)); }

// 1 / sqrt(x) for x > 0, within two units in the last place
TMPS_DEV double rsqrt64(double x) {
    if (!plain64(x) || !(__double2hiint(x) > 0)) return 1.0 / sqrt(x);
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = __fma_rn(-__dmul_rn(x, y), y, 1.0);
    return __fma_rn(__dmul_rn(y, e), __fma_rn(0.375, e, 0.5), y);
}

// root = sqrt(x): the product x / sqrt(x) corrected by its own residual; inv =
// 1 / root within two units in the last place.
TMPS_DEV void sqrt_rsqrt64(double x, double& root, double& inv) {
    if (!plain64(x) || !(__double2hiint(x) > 0)) {
        root = sqrt(x);
        inv = 1.0 / root;
        return;
    }
    inv = rsqrt64(x);
    const double g = __dmul_rn(x, inv);
    root = __fma_rn(__fma_rn(-g, g, x), __dmul_rn(0.5, inv), g);
}
// The same with inv = 1 / root.
TMPS_DEV void sqrt_rcp64(double x, double& root, double& inv) {
    sqrt_rsqrt64(x, root, inv);
    if (plain64(x)) inv = refine_rcp64(root, inv);
}
TMPS_DEV double sqrt64(double x) {
    double root, inv;
    sqrt_rsqrt64(x, root, inv);
    return root;
}
// 1 / x where y = 1 / sqrt64(x) is at hand
TMPS_DEV double rcp_of_square64(double x, double y) {
    return plain64(x) ? refine_rcp64(x, __dmul_rn(y, y)) : 1.0 / x;
}

// sqrt(s) > m, as the rounded root compares (s a sum of squares): by the high
// words of s and m * m where they differ by more than the roundings of either
// can move them, without a root.
TMPS_DEV bool root_exceeds64(double s, double m) {
    const uint32_t hs = (uint32_t)__double2hiint(s), hm = (uint32_t)__double2hiint(__dmul_rn(m, m));
    if (hs < 0x7ff00000u && hm < 0x7ff00000u && __double2hiint(m) >= 0) {
        if (hs > hm + 1u) return true;
        if (hs + 1u < hm) return false;
    }
    return sqrt64(s) > m;
}

// a * b >= 0.0, as the FP64 product compares: from the sign bits where the
// exponents keep the product clear of underflow (and neither is a NaN), the
// product itself otherwise.
TMPS_DEV bool prod_nonneg(double a, double b) {
    const int ha = __double2hiint(a), hb = __double2hiint(b);
    const int ea = (ha >> 20) & 0x7ff, eb = (hb >> 20) & 0x7ff;
    if (ea > 0x200 && ea < 0x600 && eb > 0x200 && eb < 0x600) return (ha ^ hb) >= 0;
    return a * b >= 0.0;
}

TMPS_DEV double4 ld4(const double* p, int i) { return reinterpret_cast<const double4*>(p)[i]; }
TMPS_DEV void st4(double* p, int i, double4 v) { reinterpret_cast<double4*>(p)[i] = v; }
TMPS_DEV float4 ld4f(const float* p, int i) { return reinterpret_cast<const float4*>(p)[i]; }
TMPS_DEV void st4f(float* p, int i, float4 v) { reinterpret_cast<float4*>(p)[i] = v; }

// Block-wide sum of `nv` doubles held per thread; the result lands in
// out[0..nv) of thread 0.  Fixed tree order: deterministic for a given
// block size.
template <int NV, int BLOCK>
TMPS_DEV void block_sum(double (&v)[NV], double* smem /* [NV][BLOCK/32] */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < NV; ++c) {
        double s = v[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) smem[c * (BLOCK / 32) + warp] = s;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            double s = lane < BLOCK / 32 ? smem[c * (BLOCK / 32) + lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            v[c] = s;
        }
    }
}

// Block sum of six FP64 components by halving exchanges: the FP64 pipe charges an instruction per warp however few lanes
// use it, so a shuffle tree per component (30 additions per warp) costs as
// much as several atoms' updates.  Padded to eight components, each exchange
// keeps half of what a lane holds (4 + 2 + 1 + 1 + 1 = 9 additions per
// warp), after which lane l holds component 4 b4 + 2 b3 + b2 (its lane bits
// 4, 3, 2: lane >> 2) of the warp's total.  Lanes 0..5 of warp 0 then add the warp
// totals of their component in warp order and return the block's total; the
// other threads return 0.  Fixed order: deterministic for a block size.
TMPS_DEV double warp_sum6_halving(const double (&v)[6]) {
    const int lane = threadIdx.x & 31;
    const double a[8] = {v[0], v[1], v[2], v[3], v[4], v[5], 0.0, 0.0};
    const bool b4 = (lane & 16) != 0, b3 = (lane & 8) != 0, b2 = (lane & 4) != 0;
    double r4[4], r2[2];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double send = b4 ? a[k] : a[4 + k], keep = b4 ? a[4 + k] : a[k];
        r4[k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const double send = b3 ? r4[k] : r4[2 + k], keep = b3 ? r4[2 + k] : r4[k];
        r2[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    double r = (b2 ? r2[1] : r2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? r2[0] : r2[1], 4);
    r += __shfl_xor_sync(0xffffffffu, r, 2);  // both lanes of a pair add the same two values
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    return r;
}

// `kept`: lane c < 6 holds a further value of component c; with `any` false
// (warp-uniform) every v is zero and the exchanges are left out.
template <int BLOCK>
TMPS_DEV double block_sum6_halving(const double (&v)[6], double kept, bool any,
                                                     double* smem /* [6][BLOCK / 32] */) {
    constexpr int kW = BLOCK / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double r = 0.0;
    if (any) r = __shfl_sync(0xffffffffu, warp_sum6_halving(v), (lane << 2) & 31);  // lane c < 6: component c
    if (lane < 6) smem[lane * kW + warp] = any ? r + kept : kept;
    __syncthreads();
    double t = 0.0;
    if (warp == 0 && lane < 6) {
        t = smem[lane * kW];
#pragma unroll
        for (int w = 1; w < kW; ++w) t += smem[lane * kW + w];
    }
    return t;
}

}  // namespace tmps
