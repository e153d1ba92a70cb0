// backproject_device.cuh -- device arithmetic shared by the backprojector's
// forms: the constants of the weight and of the border decisions, the asin
// and row-floor helpers, packed FP32, the output modes.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "backproject.h"

namespace ctbb {

namespace {

constexpr float kQ = 0.6f;
// slices per sub-chunk: the unit of the flat / inner / other decision
constexpr int kSub = 8;

// interp2 drops a sample when q_idx > R*nht - 2, which only the last half
// turn can reach.  Its weight still counts, so the decision is a jump in the
// image; near it the reference's own float q_idx decides.  This recomputes that
// q_idx with the reference's operations and rounding (asin through double,
// i.e. correctly rounded); it runs only when the fast coordinate is within
// kBorderBand rows of the border.
__device__ __forceinline__ bool last_turn_sample_valid(const BpParams &p, float x, float y, float theta,
                                                    float s, float c, float phat, float z, int k)
{
    float asn = (float)asin((double)__fdiv_rn(phat, p.rf));
    float ray = __fdiv_rn(__fmul_rn(p.z_rot, __fsub_rn(theta, asn)), p.two_pi);
    float lhat = __fsub_rn(__fsub_rn(__fsqrt_rn(__fsub_rn(p.rf2, __fmul_rn(phat, phat))), __fmul_rn(x, c)),
                           __fmul_rn(y, s));
    float qhat = __fdiv_rn(__fsub_rn(z, ray), __fmul_rn(lhat, p.tan_cone));
    float q_idx = __fadd_rn(__fmul_rn(__fdiv_rn(__fadd_rn(qhat, 1.0f), 2.0f), (float)p.n_rows - 1.0f),
                            (float)(k * p.n_rows));
    return !(q_idx > (float)(p.n_rows * p.nht - 2)) && !(q_idx < 0.0f);
}

constexpr float kBorderBand = 1e-3f;
// inner chunks: |q| <= kInnerMax keeps every row below R-1 after rounding;
// rows kRowMargin below the last-turn border are far from its band
constexpr float kInnerMax = 0.999f;
constexpr float kRowMargin = 0.01f;
// half-turn window margin (angle rounding is ~1e-6 half turns)
constexpr float kWindowMargin = 0.01f;

// p_idx = p / (r_f fai / 2) + 2 cc as the reference rounds it (division, then
// add), used where the interp2 border decision is close.
__device__ __forceinline__ float p_index_exact(const BpParams &p, float phat)
{
    return __fadd_rn(__fdiv_rn(phat, p.ds_half), p.two_cc);
}

// asin(a) for |a| <= 0.5 as a + a^3 P(a^2), P of degree 4 fitted here by
// weighted least squares on Chebyshev nodes (max error 0.67 ulp in float);
// larger |a| (only the corners of very wide fields) fall back to asinf.
__device__ __forceinline__ float asin_fast(float a)
{
    if (fabsf(a) > 0.5f) return asinf(a);
    float t = a * a;
    float p = fmaf(t, 0.042095037962576944f, 0.024220510033133892f);
    p = fmaf(t, p, 0.04546249911296045f);
    p = fmaf(t, p, 0.07495353339646753f);
    p = fmaf(t, p, 0.16666751488866943f);
    return fmaf(a * t, p, a);
}

// Row floors through the float unit: for |ql| < 2^22, ql + 1.5 2^23 rounded
// down is exactly 1.5 2^23 + floor(ql) (the binade [2^23, 2^24) has unit
// spacing), so one packed add gives both the floor as a float (t - 1.5 2^23,
// exact) and as an integer (the bits of t are kFloorMagicBits + floor(ql)).
// The row address is then view + bits(t) * row stride with the view's base
// moved back by kFloorMagicBits rows (64-bit modular arithmetic, folded into
// BpParams::rebin_rows on the host): one multiply-add, no conversion.
constexpr float kFloorMagic = 12582912.0f;       // 1.5 * 2^23
constexpr uint32_t kFloorMagicBits = 0x4B400000u;  // its bits
__device__ __forceinline__ float2 row_floor(float2 ql)
{
    return __fadd2_rd(ql, make_float2(kFloorMagic, kFloorMagic));
}

// Packed FP32 pairs (sm_100 family): one instruction for two lanes.
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
// Where a tile's image sums go, see backproject_column_tile.
enum { kOutScaled = 0, kOutPartial = 1, kOutFirst = 2, kOutMiddle = 3, kOutLast = 4 };

}  // namespace

}  // namespace ctbb
