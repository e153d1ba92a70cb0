// adaptive_filter.cu -- Kachelriess-Kalender adaptive raw-data filter.
//
// Reference: adaptive_filter_kk (src/preprocessing.cu:31-156) and its kernels
// (include/preprocessing.cuh:32-285), the reference's only implementation (it
// has no CPU twin; src/main.cu:222 runs it on every block).  Per pull window of
// P frames:
//   1. sup[p]      = max(0, max of frame p)                        (extract_sup)
//   2. smooth[p]   = mean of sup over an 18 deg window, clamped     (smooth_sup)
//   3. ecc[p]      = clamp(((1 - min/max) - 0.3) / 0.2, 0, 1) over a
//                    180 deg window of smooth; min/max kept         (eccentricity)
//   4. T[p]        = <= 20-step bisection between min and max so that the
//                    fraction of the 180 deg window of smooth above T matches
//                    F_MAX * strength * ecc within 1 %                (find_thresholds)
//   5. out         = 5x5x5 normalised triangle smoothing of samples > T[p],
//                    other samples copied                          (filter_projections)
// With strength 0 the stopping test divides by zero and T climbs toward the
// window maximum; samples above it are still smoothed.  That behaviour is kept.
//
// Every float operation is written as a separate rounding (__f*_rn) in the
// reference's order, so the result equals the reference kernels evaluated
// without fused multiply-adds.  GB300 mapping: step 1 is a CTA reduction per
// frame that copies the frame on the way, steps 2-3 one thread per frame, step
// 4 one warp per frame (the window counts are integers, so splitting them
// across lanes is exact), step 5 reads the frames again that hold a sample
// above their threshold and smooths those samples.  The window is so moved once
// (read and written, the HBM bound); copying after the thresholds reads it
// twice.  Every step takes a frame range, so a window whose frames arrive in
// order can be filtered as they come (AfStream).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "adaptive_filter.h"
#include "ctbb_internal.h"
#include "cuda_util.cuh"

namespace ctbb {

namespace {

constexpr float kFMax = 0.03f;  // F_MAX, include/preprocessing.cuh:23
constexpr float kPiAf = kPiBackproject;

// triangle_3d(5, i, j, k) = (3-|i-3|) + (3-|j-3|) + (3-|k-3|) + 1
// (include/preprocessing.cuh:64-67); its peak is at index 3 of 0..4.
__host__ __device__ constexpr int tri1(int i) { return 3 - (i > 3 ? i - 3 : 3 - i); }

struct AfParams {
    const float *raw;
    float *out;
    float *sup, *smooth, *ecc, *pmax, *pmin, *thr;
    float *sup_out;  // maxima to write (null: they are given)
    int P, R, N;
    int n_proj_ffs;
    int n_avg, avg_offset;
    int n_range, range_offset;
    float strength;
    int f0, f1;  // frames this launch writes: [f0, f1) of the window [0, P)
    int parts;   // af_filter_kernel: parts of a frame
};

// Groups of four consecutive samples of a frame; VEC: 16-byte accesses (whole
// groups, aligned frames).  Samples past the frame's end read 0, which no
// threshold lies below.
template <bool VEC>
__device__ __forceinline__ float4 load_group(const float *src, int i, int n)
{
    if constexpr (VEC) return __ldg(reinterpret_cast<const float4 *>(src) + i);
    float4 v;
    v.x = __ldg(src + 4 * i);
    v.y = 4 * i + 1 < n ? __ldg(src + 4 * i + 1) : 0.0f;
    v.z = 4 * i + 2 < n ? __ldg(src + 4 * i + 2) : 0.0f;
    v.w = 4 * i + 3 < n ? __ldg(src + 4 * i + 3) : 0.0f;
    return v;
}

template <bool VEC>
__device__ __forceinline__ void store_group(float *dst, int i, int n, float4 v)
{
    if constexpr (VEC) {
        reinterpret_cast<float4 *>(dst)[i] = v;
    } else {
        dst[4 * i] = v.x;
        if (4 * i + 1 < n) dst[4 * i + 1] = v.y;
        if (4 * i + 2 < n) dst[4 * i + 2] = v.z;
        if (4 * i + 3 < n) dst[4 * i + 3] = v.w;
    }
}

// Step 1, and the copy of every sample that step 5 does not change: one CTA
// per frame, last frame first (the rebinning starts with the first, which L2
// then still holds), kCopyUnroll groups in flight per thread.  Bound by HBM:
// 11 264 frames of 736 x 32 (1.06 GB each way) in 300 us, 7.1 TB/s.  The maxima
// and the copy as separate passes: 146 + 365 us.  Eight CTAs per SM, unrolls of
// 2 and 8 and streaming loads or stores are within 3 % or slower.
constexpr int kCopyUnroll = 4;

template <bool VEC>
__global__ void __launch_bounds__(256, 4) af_copy_kernel(AfParams p)
{
    const int proj = p.f1 - 1 - (int)blockIdx.x;
    const size_t frame = (size_t)p.R * p.N;
    const float *src = p.raw + (size_t)proj * frame;
    float *dst = p.out + (size_t)proj * frame;
    const int n = (int)frame, n4 = (n + 3) / 4;
    float m = 0.0f;
    for (int i0 = threadIdx.x; i0 < n4; i0 += kCopyUnroll * 256) {
        float4 v[kCopyUnroll];
#pragma unroll
        for (int u = 0; u < kCopyUnroll; ++u) {
            const int i = i0 + u * 256;
            v[u] = i < n4 ? load_group<VEC>(src, i, n) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int u = 0; u < kCopyUnroll; ++u) {
            const int i = i0 + u * 256;
            if (i < n4) store_group<VEC>(dst, i, n, v[u]);
            m = fmaxf(fmaxf(m, fmaxf(v[u].x, v[u].y)), fmaxf(v[u].z, v[u].w));
        }
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < 8 ? red[threadIdx.x] : 0.0f;
        for (int o = 4; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0 && p.sup_out) p.sup_out[proj] = m;
    }
}

// STAGED: the CTA's windows, weighted, in shared memory (kSmoothSmem); an
// averaging window past that (more than 12 161 frames) is read as it lies.  The sum
// keeps the reference's order in both.
constexpr size_t kSmoothSmem = 48 * 1024;

__host__ __device__ constexpr size_t smooth_smem(int n_avg) { return (size_t)(127 + (size_t)n_avg) * sizeof(float); }

template <bool STAGED>
__global__ void af_smooth_kernel(AfParams p)
{
    extern __shared__ float win[];
    const int first = p.f0 + blockIdx.x * blockDim.x, n = min((int)blockDim.x, p.f1 - first);
    const float w = __fdiv_rn(1.0f, (float)p.n_avg);
    const int max_idx = p.P - 1;
    auto weighted = [&](int i) { return __fmul_rn(w, p.sup[min(max(first - p.avg_offset + i, 0), max_idx)]); };
    if (STAGED) {
        for (int i = threadIdx.x; i < n + p.n_avg - 1; i += blockDim.x) win[i] = weighted(i);
        __syncthreads();
    }
    if ((int)threadIdx.x >= n) return;
    float acc = 0.0f;
#pragma unroll 8
    for (int i = 0; i < p.n_avg; i++)
        acc = __fadd_rn(acc, STAGED ? win[threadIdx.x + i] : weighted((int)threadIdx.x + i));
    p.smooth[first + threadIdx.x] = acc;
}

// eccentricity from the window's extremes (include/preprocessing.cuh:133-150)
__device__ __forceinline__ void write_ecc(const AfParams &p, int proj, float vmax, float vmin)
{
    p.pmax[proj] = vmax;
    p.pmin[proj] = vmin;
    float e = __fsub_rn(1.0f, __fdiv_rn(vmin, vmax));
    e = __fdiv_rn(__fsub_rn(e, 0.3f), __fsub_rn(0.5f, 0.3f));
    float out;
    if (e > 1) out = 1.0f;
    else if (e < 0) out = 0.0f;
    else out = e;
    p.ecc[proj] = out;
}

// Extremes of every frame's window by doubling: after the pass of length len,
// hi[i] is the maximum of len consecutive means from i (lo the minimum), and a
// window is the union of two such runs.  Extremes do not depend on the order,
// so this equals the reference's scan of the window (max from 0, min from
// 10000, frames outside the scan repeated at its ends).  Instead of 2305
// reads per frame (config 2), 12 passes over the CTA's 2560 means: 62 -> 9 us
// for 11 264 frames.
constexpr int kEccFrames = 256;
constexpr size_t kEccSmem = 48 * 1024;

__host__ __device__ constexpr size_t ecc_smem(int n_range)
{
    return 4 * sizeof(float) * (size_t)(kEccFrames + n_range - 1);
}

__global__ void __launch_bounds__(kEccFrames) af_ecc_kernel(AfParams p)
{
    extern __shared__ float win[];
    const int first = p.f0 + blockIdx.x * kEccFrames, n = min(kEccFrames, p.f1 - first);
    const int w = n + p.n_range - 1, stride = kEccFrames + p.n_range - 1;
    float *hi = win, *lo = win + stride, *hi2 = win + 2 * stride, *lo2 = win + 3 * stride;
    for (int i = threadIdx.x; i < w; i += kEccFrames) {
        const int idx = first - p.range_offset + i;
        const bool in = idx >= 0 && idx < p.P;  // a window past an end holds the end frame itself
        const float v = in ? p.smooth[idx] : 0.0f;
        hi[i] = fmaxf(v, 0.0f);
        lo[i] = in ? fminf(v, 10000.0f) : 10000.0f;
    }
    __syncthreads();
    int len = 1;
    for (; 2 * len <= p.n_range; len *= 2) {
        for (int i = threadIdx.x; i + 2 * len <= w; i += kEccFrames) {
            hi2[i] = fmaxf(hi[i], hi[i + len]);
            lo2[i] = fminf(lo[i], lo[i + len]);
        }
        __syncthreads();
        float *t = hi;
        hi = hi2;
        hi2 = t;
        t = lo;
        lo = lo2;
        lo2 = t;
    }
    const int i = threadIdx.x, j = i + p.n_range - len;
    if (i < n) write_ecc(p, first + i, fmaxf(hi[i], hi[j]), fminf(lo[i], lo[j]));
}

// The same with one thread reading its whole window, for windows past the
// shared memory of the kernel above (turns of more than 5600 frames).
__global__ void af_ecc_long_kernel(AfParams p)
{
    int proj = p.f0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (proj >= p.f1) return;
    int max_idx = p.P - 1;
    float vmax = 0.0f, vmin = 10000.0f;
    for (int i = 0; i < p.n_range; i++) {
        int idx = proj - p.range_offset + i;
        idx = idx < 0 ? 0 : (idx > max_idx ? max_idx : idx);
        float v = p.smooth[idx];
        if (v > vmax) vmax = v;
        if (v < vmin) vmin = v;
    }
    write_ecc(p, proj, vmax, vmin);
}

// Step 4: the reference's bisection, one warp per frame.  STAGED: the window of
// a CTA's frames is in shared memory with the extremes of each 32 means, so a
// count above T reads only the few chunks that T cuts through -- the means are
// 18 degree averages, so a chunk is narrow -- and once 256 values lie between
// the bounds they move to registers.  11 264 frames of 2305: 70 us with the
// window in registers and every count over all of it, 43 us so (4446 and 3250
// instructions a frame, and the chain of a bisection's steps).  Otherwise a
// window of up to 256 means is in registers from the start (192 views a turn:
// 2 us faster than staged), and one beyond kThrSmem counts from global memory.
constexpr int kThrFrames = 8;  // frames (warps) per CTA
constexpr int kFew = 8;        // values per lane once few are left
constexpr size_t kThrSmem = 48 * 1024;

__host__ __device__ constexpr int thr_chunks(int n_range) { return (n_range + kThrFrames - 1 + 31) / 32; }
__host__ __device__ constexpr size_t thr_smem(int n_range)
{
    return sizeof(float) * ((size_t)thr_chunks(n_range) * (32 + 2) + kThrFrames * 32 * kFew);
}

template <bool STAGED>
__global__ void __launch_bounds__(32 * kThrFrames) af_threshold_kernel(AfParams p)
{
    extern __shared__ float win[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = p.f0 + (int)blockIdx.x * kThrFrames, proj = first + warp;
    // the CTA's window and this frame's, cut at the scan's ends
    const int cta_begin = max(first - p.range_offset, 0);
    const int begin = max(proj - p.range_offset, 0);
    const int numel = min(proj - p.range_offset + p.n_range, p.P) - begin;
    float *lo = win + 32 * thr_chunks(p.n_range), *hi = lo + thr_chunks(p.n_range);
    float *kept = hi + thr_chunks(p.n_range) + warp * (32 * kFew);
    if (STAGED) {
        const int last = min(first + kThrFrames, p.f1) - 1;
        const int len = min(last - p.range_offset + p.n_range, p.P) - cta_begin;
        for (int c = warp; 32 * c < len; c += kThrFrames) {
            const float v = 32 * c + lane < len ? p.smooth[cta_begin + 32 * c + lane] : 0.0f;
            win[32 * c + lane] = v;
            // means are never negative: their bits order as they do
            const unsigned least = __reduce_min_sync(0xffffffffu, __float_as_uint(v));
            const unsigned most = __reduce_max_sync(0xffffffffu, __float_as_uint(v));
            if (lane == 0) {
                lo[c] = __uint_as_float(least);
                hi[c] = __uint_as_float(most);
            }
        }
        __syncthreads();
    }
    if (proj >= p.f1) return;
    const int w0 = begin - cta_begin, w1 = w0 + numel;  // this frame's window in `win`
    const int c1 = (w1 + 31) / 32;
    int above = 0;  // values no longer kept that are above every further threshold
    bool is_few = false;
    float v[kFew];  // a value not kept is -inf, never above a threshold
    if (!STAGED && numel <= 32 * kFew) {
#pragma unroll
        for (int k = 0; k < kFew; ++k) v[k] = lane + 32 * k < numel ? p.smooth[begin + lane + 32 * k] : -INFINITY;
        is_few = true;
    }
    auto count = [&](float T) {
        int n = 0;
        if (is_few) {
#pragma unroll
            for (int k = 0; k < kFew; ++k) n += v[k] > T ? 1 : 0;
        } else if (STAGED) {
            for (int base = w0 / 32; base < c1; base += 32) {
                const int c = base + lane;
                const bool some = c < c1 && hi[min(c, c1 - 1)] > T;
                const bool all = some && lo[c] > T && 32 * c >= w0 && 32 * c + 32 <= w1;
                n += all ? 32 : 0;
                for (unsigned m = __ballot_sync(0xffffffffu, some && !all); m; m &= m - 1) {
                    const int i = 32 * (base + __ffs(m) - 1) + lane;
                    n += i >= w0 && i < w1 && win[i] > T ? 1 : 0;
                }
            }
        } else {
            for (int i = lane; i < numel; i += 32) n += p.smooth[begin + i] > T ? 1 : 0;
        }
        return __reduce_add_sync(0xffffffffu, n) + above;
    };
    const float inv_pi = 1.0f / kPiAf, inv_turn = __fdiv_rn(1.0f, (float)p.n_proj_ffs);
    auto fraction = [&](int n) { return __fmul_rn(__fmul_rn(inv_pi, (float)n), inv_turn); };
    float lower = p.pmin[proj], upper = p.pmax[proj];
    int n_lower = numel, n_upper = 0;  // values above each bound (at most, for the first)
    float T = __fdiv_rn(__fadd_rn(upper, lower), 2.0f);
    const float lhs = __fmul_rn(__fmul_rn(kFMax, p.strength), p.ecc[proj]);
    int n = count(T);
    float rhs = fraction(n);
    int iter = 0;
    // the reference compares the float quotient, promoted to double, with
    // 0.01; no float lies between 0.01f and 0.01
    while (__fdiv_rn(fabsf(__fsub_rn(lhs, rhs)), lhs) > 0.01f) {
        if (iter >= 20) break;
        iter += 1;
        if (rhs > lhs) {
            lower = T;
            n_lower = n;
        } else if (rhs < lhs) {
            upper = T;
            n_upper = n;
        } else {
            break;
        }
        if (STAGED && !is_few && n_lower - n_upper <= 32 * kFew) {
            int at = 0;
            for (int base = w0 / 32; base < c1; base += 32) {
                const int c = base + lane;
                const bool some = c < c1 && hi[min(c, c1 - 1)] > lower && lo[min(c, c1 - 1)] <= upper;
                for (unsigned m = __ballot_sync(0xffffffffu, some); m; m &= m - 1) {
                    const int i = 32 * (base + __ffs(m) - 1) + lane;
                    const float x = win[i];
                    const bool keep = i >= w0 && i < w1 && x > lower && x <= upper;
                    const unsigned who = __ballot_sync(0xffffffffu, keep);
                    if (keep) kept[at + __popc(who & ((1u << lane) - 1u))] = x;
                    at += __popc(who);
                }
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < kFew; ++k) v[k] = lane + 32 * k < at ? kept[lane + 32 * k] : -INFINITY;
            above = n_upper;
            is_few = true;
        }
        T = __fdiv_rn(__fadd_rn(lower, upper), 2.0f);
        n = count(T);
        rhs = fraction(n);
    }
    if (lane == 0) p.thr[proj] = T;
}

// 5x5x5 triangle smoothing of up to kWarpSamples listed samples (frame, sample
// of the frame) by a warp, taps added in the reference's order (channel, row,
// frame).  The lanes fetch all taps at once into shared memory, one tap of
// every sample per kWarpSamples lanes, and a lane then adds its sample's; a
// thread that fetched its own sample's taps waited for them five times, and a
// list is often shorter than a warp.  A tap out of range counts as 0, which
// leaves the sum as it is; norm is the exact integer sum of the weights in
// range.
constexpr int kWarpSamples = 4;

__device__ __forceinline__ void smooth_samples(const AfParams &p, const int2 *list, int n, float *taps)
{
    const int lane = threadIdx.x & 31, s = lane % kWarpSamples;
    const size_t frame = (size_t)p.R * p.N;
    const int2 at = list[min(s, n - 1)];
    const int gp = at.x, gr = at.y / p.N, gc = at.y - gr * p.N;
    constexpr int kTapLanes = 32 / kWarpSamples, kFetch = (125 + kTapLanes - 1) / kTapLanes;
    float x[kFetch];
#pragma unroll
    for (int m = 0; m < kFetch; ++m) {
        const int tap = lane / kWarpSamples + kTapLanes * m;
        const int c = gc + tap / 25 - 2, r = gr + tap / 5 % 5 - 2, f = gp + tap % 5 - 2;
        const bool in = tap < 125 && c >= 0 && c < p.N && r >= 0 && r < p.R && f >= 0 && f < p.P;
        x[m] = in ? __ldg(p.raw + (size_t)f * frame + (size_t)r * p.N + c) : 0.0f;
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < kFetch; ++m)
        if (lane / kWarpSamples + kTapLanes * m < 125) taps[lane + 32 * m] = x[m];
    __syncwarp();
    if (lane < min(n, kWarpSamples)) {
        int ni = 0, nj = 0, nk = 0, si = 0, sj = 0, sk = 0;
#pragma unroll
        for (int d = 0; d < 5; ++d) {
            if (gc + d - 2 >= 0 && gc + d - 2 < p.N) { ni++; si += tri1(d); }
            if (gr + d - 2 >= 0 && gr + d - 2 < p.R) { nj++; sj += tri1(d); }
            if (gp + d - 2 >= 0 && gp + d - 2 < p.P) { nk++; sk += tri1(d); }
        }
        const float norm = (float)(nj * nk * si + ni * nk * sj + ni * nj * sk + ni * nj * nk);
        float val = 0.0f;
#pragma unroll
        for (int t = 0; t < 125; ++t)
            val = __fadd_rn(val, __fmul_rn(taps[kWarpSamples * t + lane],
                                           (float)(tri1(t / 25) + tri1(t / 5 % 5) + tri1(t % 5) + 1)));
        p.out[(size_t)gp * frame + at.y] = __fmul_rn(__fdiv_rn(1.0f, norm), val);
    }
}

// The same for a part of a frame, rows [row0, row1), that is dense in samples
// above the threshold: tiles of kTileRows x kTileCols outputs with their halo
// in shared memory, a thread for four consecutive channels of a row, so that a
// tap fetched serves up to four sums (50 reads of shared memory per sample
// instead of 125).  Column c of a tile row lies at (c mod 4, c / 4): lanes four
// channels apart read consecutive words.  Every thread of the CTA calls it;
// true if about a sixteenth of the part or more was above.
constexpr int kTileRows = 4, kTileCols = 256;  // a warp per half row
constexpr int kPlane = 68;  // (kTileCols + 4) / 4 words, rounded up against store conflicts
constexpr int kTileRow = 4 * kPlane, kTileFrame = (kTileRows + 4) * kTileRow, kTileFloats = 5 * kTileFrame;

__device__ __forceinline__ bool smooth_part(const AfParams &p, int f, float T, int row0, int row1, float *tile)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t frame = (size_t)p.R * p.N;
    bool any = false, held = false;
    for (int r0 = row0; r0 < row1; r0 += kTileRows)
        for (int c0 = 0; c0 < p.N; c0 += kTileCols) {
            const int n_rows = min(kTileRows, row1 - r0) + 4;
            __syncthreads();  // the last tile is read
            for (int q = warp; q < 5 * n_rows; q += 8) {
                const int k = q / n_rows, tr = q - k * n_rows, gf = f + k - 2, gr = r0 + tr - 2;
                const bool in = gf >= 0 && gf < p.P && gr >= 0 && gr < p.R;
                const float *src = p.raw + (in ? (size_t)gf * frame + (size_t)gr * p.N : 0);
                float *dst = tile + k * kTileFrame + tr * kTileRow + (lane & 3) * kPlane + (lane >> 2);
                float x[(kTileCols + 4 + 31) / 32];
#pragma unroll
                for (int m = 0; m < (kTileCols + 4 + 31) / 32; ++m) {
                    const int gc = c0 + lane + 32 * m - 2;
                    x[m] = in && lane + 32 * m < kTileCols + 4 && gc >= 0 && gc < p.N ? __ldg(src + gc) : 0.0f;
                }
#pragma unroll
                for (int m = 0; m < (kTileCols + 4 + 31) / 32; ++m)
                    if (lane + 32 * m < kTileCols + 4) dst[8 * m] = x[m];
            }
            __syncthreads();
            const int tr = warp & 3, tc = 32 * (warp >> 2) + lane, gr = r0 + tr, gc = c0 + 4 * tc;
            if (gr >= row1 || gc >= p.N) continue;
            const float *at = tile + tr * kTileRow + tc;
            float x[4], val[4] = {};
#pragma unroll
            for (int t = 0; t < 8; ++t) {  // channel gc + t - 2
                float v[25];
#pragma unroll
                for (int m = 0; m < 25; ++m)
                    v[m] = at[(m % 5) * kTileFrame + (m / 5) * kTileRow + (t & 3) * kPlane + (t >> 2)];
                if (t >= 2 && t < 6) x[t - 2] = v[12];
#pragma unroll
                for (int o = 0; o < 4; ++o)
                    if (t - o >= 0 && t - o < 5) {
#pragma unroll
                        for (int m = 0; m < 25; ++m)
                            val[o] = __fadd_rn(val[o], __fmul_rn(v[m], (float)(tri1(t - o) + tri1(m / 5) + tri1(m % 5) + 1)));
                    }
            }
            held = true;
            int nj = 0, nk = 0, sj = 0, sk = 0;
#pragma unroll
            for (int d = 0; d < 5; ++d) {
                if (gr + d - 2 >= 0 && gr + d - 2 < p.R) { nj++; sj += tri1(d); }
                if (f + d - 2 >= 0 && f + d - 2 < p.P) { nk++; sk += tri1(d); }
            }
#pragma unroll
            for (int o = 0; o < 4; ++o) {
                const int c = gc + o;
                if (c >= p.N || !(x[o] > T)) continue;
                any = true;
                int ni = 0, si = 0;
#pragma unroll
                for (int d = 0; d < 5; ++d)
                    if (c + d - 2 >= 0 && c + d - 2 < p.N) { ni++; si += tri1(d); }
                const float norm = (float)(nj * nk * si + ni * nk * sj + ni * nj * sk + ni * nj * nk);
                p.out[(size_t)f * frame + (size_t)gr * p.N + c] = __fmul_rn(__fdiv_rn(1.0f, norm), val[o]);
            }
        }
    // half of the threads with a sample of theirs above, at a dozen samples each
    return 2 * __syncthreads_count(any) >= __syncthreads_count(held);
}

// Step 5, on a copy of the frames (af_copy_kernel): only frames whose maximum
// exceeds their threshold are read again (thresholds lie between means of
// maxima, so they are never negative), one in twenty at strength 1.  They come
// in short runs, so a frame is cut into up to kParts parts, and each CTA serves
// one part of every `lanes`-th frame: it lists the samples above the threshold
// in shared memory, over all its frames, and smooths them together, or earlier
// when the list runs full.  Bound by the waits of its chain (thresholds, four
// rounds of loads at a time, taps): 42 us for the window above, where a CTA per
// frame with a thread per listed sample took 69 us; 4 or 16 parts take 2 %
// longer for the call, 8 rounds at a time 4 %.
// A warp smooths four listed samples at a time, which a part with many leaves
// to smooth_part: when the list fills up and a sixteenth of the part at hand
// is in it, that part and those after it are smoothed as tiles, until one is
// not dense (a listed sample costs some sixteen times a tile's).  2816 frames
// of 736 x 32 with 90 % of the samples above: 15.3 ms all from the list, 1.44
// so; of 738 x 32 14.7 and 1.44 (1.53 when every sample went through a tile);
// with 3 % above 0.78 and 0.51.
constexpr int kParts = 8;
constexpr int kAhead = 4;
constexpr int kListRoom = 4 * 256;  // samples a round can add, and the fewest of a part
constexpr int kSmoothListMax = 2 * kListRoom;
constexpr int kFilterCtas = 2;

template <bool VEC>
__global__ void __launch_bounds__(256, kFilterCtas) af_filter_kernel(AfParams p)
{
    // the list and the warps' taps, or a tile
    constexpr int kTaps = 125 * kWarpSamples;
    static_assert(2 * kSmoothListMax + 8 * kTaps <= kTileFloats, "the list and the taps lie in the tile's place");
    __shared__ __align__(16) float work[kTileFloats];
    int2 *list = reinterpret_cast<int2 *>(work);
    float *taps = work + 2 * kSmoothListMax + threadIdx.x / 32 * kTaps;
    __shared__ int active[256];
    __shared__ float active_thr[256];
    __shared__ int n_list, n_active, part_at;
    const int part = blockIdx.x % p.parts, lanes = gridDim.x / p.parts;
    const size_t frame = (size_t)p.R * p.N;
    const int n_frame = (int)frame, n4 = (n_frame + 3) / 4;
    // a part is a number of rows, all but the last part's a multiple of 4 (whole
    // groups, and whole tiles)
    const int rows4 = (p.R + 3) / 4, row0 = 4 * (part * rows4 / p.parts);
    const int row1 = min(4 * ((part + 1) * rows4 / p.parts), p.R);
    const int g0 = row0 / 4 * p.N, g1 = row1 < p.R ? row1 / 4 * p.N : n4;
    auto smooth_listed = [&](int n) {
        for (int j = (int)threadIdx.x / 32 * kWarpSamples; j < n; j += 8 * kWarpSamples)
            smooth_samples(p, list + j, n - j, taps);
    };
    bool dense = false;  // the last part was; the list is empty
    if (threadIdx.x == 0) n_list = 0;
    for (int first = p.f0 + (int)blockIdx.x / p.parts; first < p.f1; first += 256 * lanes) {
        if (threadIdx.x == 0) n_active = 0;
        __syncthreads();
        const int f = first + (int)threadIdx.x * lanes;
        const float T = f < p.f1 ? __ldg(p.thr + f) : 0.0f;
        if (f < p.f1 && __ldg(p.sup + f) > T) {
            const int slot = atomicAdd(&n_active, 1);
            active[slot] = f;
            active_thr[slot] = T;
        }
        __syncthreads();
        const int n = n_active;
        // rounds of 256 groups, the loads of kAhead of them in flight
        const int rounds = (g1 - g0 + 255) / 256;
        for (int w0 = 0, w1; w0 < n * rounds; w0 = w1) {
            if (dense) {  // w0 is the first round of a part
                const int a = w0 / rounds;
                dense = smooth_part(p, active[a], active_thr[a], row0, row1, work);
                w1 = w0 + rounds;
                continue;
            }
            w1 = w0 + kAhead;
            float4 v[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const int a = (w0 + u) / rounds, i = g0 + (w0 + u - a * rounds) * 256 + (int)threadIdx.x;
                v[u] = a < n && i < g1 ? load_group<VEC>(p.raw + (size_t)active[a] * frame, i, n_frame)
                                       : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const int a = (w0 + u) / rounds, round = w0 + u - a * rounds, i = g0 + round * 256 + (int)threadIdx.x;
                if (a >= n) break;
                const float T = active_thr[a];
                int last = 0;
                if (v[u].x > T || v[u].y > T || v[u].z > T || v[u].w > T) {
                    const float c[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (c[e] > T) {
                            last = atomicAdd(&n_list, 1);
                            list[last] = make_int2(active[a], 4 * i + e);
                        }
                }
                // a slot of the list's second half was taken: the next round may not fit
                if (__syncthreads_or(last >= kListRoom)) {
                    // this part's samples are the list's last
                    const int listed = n_list;
                    for (int j = threadIdx.x; j < listed; j += 256)
                        if (list[j].x == active[a] && (j == 0 || list[j - 1].x != active[a])) part_at = j;
                    __syncthreads();
                    dense = 4 * (listed - part_at) >= min(g0 + (round + 1) * 256, g1) - g0;
                    smooth_listed(dense ? part_at : listed);
                    __syncthreads();
                    if (threadIdx.x == 0) n_list = 0;
                    __syncthreads();
                    if (dense) {
                        w1 = a * rounds;
                        break;
                    }
                }
            }
        }
        __syncthreads();  // `active` and its count are read before they are written again
    }
    __syncthreads();
    smooth_listed(n_list);
}

// One thread per frame of the window: can this window's filtered frame
// differ from the larger window's?  Not when no sample exceeds either
// threshold (every sample is at most the frame's maximum sup), and not when
// the thresholds agree and the smoothing stencil does not reach past this
// window's ends where the larger window goes on.  NaN thresholds count as
// differing.
__global__ void af_dirty_kernel(const float *sup, const float *thr_union, const float *thr, int P, int fa, int fb,
                                int lo_edge, int hi_edge, unsigned char *dirty)
{
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= P) return;
    unsigned char d = 0;
    if (f < fa || f >= fb) {
        const float s = sup[f], tb = thr[f], tu = thr_union[f];
        const bool end = (lo_edge && f < 2) || (hi_edge && f >= P - 2);
        const bool same = (s <= tb && s <= tu) || (tb == tu && !end);
        d = same ? 0 : 1;
    }
    dirty[f] = d;
}

}  // namespace

size_t adaptive_filter_scratch_floats(size_t n_proj_pull) { return 6 * n_proj_pull; }

namespace {

int af_params(const struct recon_metadata &mr, const float *d_in, float *d_out, float *d_scratch, AfParams *pp)
{
    AfParams &p = *pp;
    p.raw = d_in;
    p.out = d_out;
    p.P = (int)mr.ri.n_proj_pull;
    p.R = (int)mr.cg.n_rows_raw;
    p.N = (int)mr.cg.n_channels;
    p.n_proj_ffs = (int)mr.cg.n_proj_ffs;
    p.sup = d_scratch;
    p.smooth = d_scratch + p.P;
    p.ecc = d_scratch + 2 * (size_t)p.P;
    p.pmax = d_scratch + 3 * (size_t)p.P;
    p.pmin = d_scratch + 4 * (size_t)p.P;
    p.thr = d_scratch + 5 * (size_t)p.P;
    // window sizes, include/preprocessing.cuh:92-96 and :119-122
    int n_avg = (int)ceilf((18.0f / 360.0f) * (float)p.n_proj_ffs);
    n_avg = n_avg + (1 - n_avg % 2);
    p.n_avg = n_avg;
    p.avg_offset = (int)floorf((float)(n_avg / 2));
    int n_range = (int)ceilf((180.0f / 360.0f) * (float)p.n_proj_ffs);
    n_range = n_range + (1 - n_range % 2);
    p.n_range = n_range;
    p.range_offset = (int)floorf((float)(n_range / 2));
    p.strength = mr.rp.adaptive_filtration_s;
    p.sup_out = nullptr;
    p.f0 = 0;
    p.f1 = p.P;
    p.parts = 1;
    if (p.P <= 0 || p.R <= 0 || p.N <= 0) {
        set_error("adaptive filter: empty pull window");
        return CTBB_ERR_ARGUMENT;
    }
    return CTBB_OK;
}

// The five steps over frame ranges: maxima (and the copy) of [sup0, sup1),
// moving means of [smooth0, smooth1), eccentricity and threshold of [thr0,
// thr1), smoothing of [out0, out1).  `copied`: the frames of the last range
// went through the first step with this p.out; otherwise the last step copies
// them too.  Each range may be empty; a step reads the earlier steps' results
// of the frames its windows cover, which the caller has launched before.
int af_launch(AfParams p, int sup0, int sup1, int smooth0, int smooth1, int thr0, int thr1, int out0, int out1,
              bool copied, cudaStream_t stream)
{
    int launches = 0;
    // frames start 16-byte aligned: whole groups of four
    const bool vec = (size_t)p.R * p.N % 4 == 0 &&
                     (reinterpret_cast<uintptr_t>(p.raw) | reinterpret_cast<uintptr_t>(p.out)) % 16 == 0;
    if (sup1 > sup0) {
        p.f0 = sup0;
        p.f1 = sup1;
        p.sup_out = p.sup;
        if (vec) af_copy_kernel<true><<<sup1 - sup0, 256, 0, stream>>>(p);
        else af_copy_kernel<false><<<sup1 - sup0, 256, 0, stream>>>(p);
        ++launches;
    }
    if (smooth1 > smooth0) {
        p.f0 = smooth0;
        p.f1 = smooth1;
        const int ctas = (smooth1 - smooth0 + 127) / 128;
        if (smooth_smem(p.n_avg) <= kSmoothSmem)
            af_smooth_kernel<true><<<ctas, 128, smooth_smem(p.n_avg), stream>>>(p);
        else
            af_smooth_kernel<false><<<ctas, 128, 0, stream>>>(p);
        ++launches;
    }
    if (thr1 > thr0) {
        int n = thr1 - thr0;
        p.f0 = thr0;
        p.f1 = thr1;
        if (ecc_smem(p.n_range) <= kEccSmem)
            af_ecc_kernel<<<(n + kEccFrames - 1) / kEccFrames, kEccFrames, ecc_smem(p.n_range), stream>>>(p);
        else
            af_ecc_long_kernel<<<(n + 127) / 128, 128, 0, stream>>>(p);
        const int ctas = (n + kThrFrames - 1) / kThrFrames;
        if (p.n_range > 32 * kFew && thr_smem(p.n_range) <= kThrSmem)
            af_threshold_kernel<true><<<ctas, 32 * kThrFrames, thr_smem(p.n_range), stream>>>(p);
        else
            af_threshold_kernel<false><<<ctas, 32 * kThrFrames, 0, stream>>>(p);
        launches += 2;
    }
    if (out1 > out0) {
        const int n = out1 - out0;
        p.f0 = out0;
        p.f1 = out1;
        if (!copied) {
            p.sup_out = nullptr;
            if (vec) af_copy_kernel<true><<<n, 256, 0, stream>>>(p);
            else af_copy_kernel<false><<<n, 256, 0, stream>>>(p);
            ++launches;
        }
        p.parts = (int)std::min<size_t>(std::min(kParts, (p.R + 3) / 4),
                                        std::max<size_t>(1, (size_t)p.R * p.N / kListRoom));
        const int grid = p.parts * std::min(n, std::max(1, num_sms() * kFilterCtas / p.parts));
        if (vec) af_filter_kernel<true><<<grid, 256, 0, stream>>>(p);
        else af_filter_kernel<false><<<grid, 256, 0, stream>>>(p);
        launches += 1;
    }
    count_launch(launches);
    CTBB_CUDA_TRY(cudaGetLastError());
    return CTBB_OK;
}

}  // namespace

int launch_adaptive_filter(const struct recon_metadata &mr, const float *d_in, float *d_out,
                           float *d_scratch, cudaStream_t stream)
{
    AfParams p;
    CTBB_TRY(af_params(mr, d_in, d_out, d_scratch, &p));
    return af_launch(p, 0, p.P, 0, p.P, 0, p.P, 0, p.P, true, stream);
}

int adaptive_filter_edge_reach(const struct recon_metadata &mr)
{
    AfParams p;
    float dummy = 0.0f;
    if (af_params(mr, &dummy, &dummy, &dummy, &p) != CTBB_OK) return 0;
    return p.range_offset + p.avg_offset;
}

int launch_adaptive_filter_ends_thresholds(const struct recon_metadata &mr, const float *d_in, const float *d_sup,
                                           float *d_scratch, int fa, int fb, cudaStream_t stream)
{
    AfParams p;
    CTBB_TRY(af_params(mr, d_in, nullptr, d_scratch, &p));
    p.sup = const_cast<float *>(d_sup);  // read only: no maxima are launched
    fa = std::min(std::max(fa, 0), p.P);
    fb = std::min(std::max(fb, fa), p.P);
    CTBB_TRY(af_launch(p, 0, 0, 0, p.P, 0, fa, 0, 0, false, stream));
    return af_launch(p, 0, 0, 0, 0, fb, p.P, 0, 0, false, stream);
}

int launch_adaptive_filter_dirty(const struct recon_metadata &mr, const float *d_sup, const float *d_thr_union,
                                 const float *d_scratch, int fa, int fb, int lo_edge, int hi_edge,
                                 unsigned char *d_dirty, cudaStream_t stream)
{
    AfParams p;
    float dummy = 0.0f;
    CTBB_TRY(af_params(mr, &dummy, &dummy, const_cast<float *>(d_scratch), &p));
    fa = std::min(std::max(fa, 0), p.P);
    fb = std::min(std::max(fb, fa), p.P);
    af_dirty_kernel<<<(p.P + 255) / 256, 256, 0, stream>>>(d_sup, d_thr_union, p.thr, p.P, fa, fb, lo_edge,
                                                              hi_edge, d_dirty);
    count_launch(1);
    CTBB_CUDA_TRY(cudaGetLastError());
    return CTBB_OK;
}

int launch_adaptive_filter_output(const struct recon_metadata &mr, const float *d_in, float *d_out,
                                  const float *d_sup, float *d_scratch, int f0, int f1, cudaStream_t stream)
{
    AfParams p;
    CTBB_TRY(af_params(mr, d_in, d_out, d_scratch, &p));
    p.sup = const_cast<float *>(d_sup);
    f0 = std::min(std::max(f0, 0), p.P);
    f1 = std::min(std::max(f1, f0), p.P);
    return af_launch(p, 0, 0, 0, 0, 0, 0, f0, f1, false, stream);
}

AfStream::AfStream(const struct recon_metadata &mr) : P((int)mr.ri.n_proj_pull)
{
    int n_proj_ffs = (int)mr.cg.n_proj_ffs;
    int n_avg = (int)ceilf((18.0f / 360.0f) * (float)n_proj_ffs);
    n_avg = n_avg + (1 - n_avg % 2);
    int n_range = (int)ceilf((180.0f / 360.0f) * (float)n_proj_ffs);
    n_range = n_range + (1 - n_range % 2);
    avg_reach = n_avg / 2;
    range_reach = n_range / 2;
}

int AfStream::advance(const struct recon_metadata &mr, const float *d_in, float *d_out, float *d_scratch,
                      int arrived, cudaStream_t stream)
{
    AfParams p;
    CTBB_TRY(af_params(mr, d_in, d_out, d_scratch, &p));
    arrived = std::min(arrived, P);
    bool all = arrived == P;
    // a moving mean needs the maxima up to avg_reach frames ahead, the
    // eccentricity and threshold the means up to range_reach ahead, the
    // smoothing the thresholds and raw frames of +-2 frames
    int smoothed = all ? P : std::max(0, arrived - avg_reach);
    int finished = all ? P : std::max(0, std::min(smoothed - range_reach, arrived - 2));
    smoothed = std::max(smoothed, n_smoothed);
    finished = std::max(finished, n_filtered);
    CTBB_TRY(af_launch(p, n_sup, arrived, n_smoothed, smoothed, n_filtered, finished, n_filtered, finished, true,
                       stream));
    n_sup = std::max(n_sup, arrived);
    n_smoothed = smoothed;
    n_filtered = finished;
    return CTBB_OK;
}

}  // namespace ctbb

// --------------------------------------------------------------------------
// Adaptive filter without any allocation
// --------------------------------------------------------------------------
//
// For callers that must not allocate device memory while a scan is being
// processed -- a scanner-side service that reserves all device memory at
// start-up and keeps cudaMalloc (which can synchronise the whole device and
// has unbounded latency) out of its per-scan path, or a host process whose
// device memory belongs to another allocator (a framework's caching pool, a
// fixed MPS/MIG quota) -- this variant takes its per-frame statistics from a
// fixed array in the library's static device memory instead of the library's
// allocated workspace.  The caller still passes the input and output buffers.

namespace ctbb {

// Largest pull window (frames) the static scratch holds; config-3 blocks pull
// 8448 frames and config-2 blocks 11264.
constexpr size_t kNoAllocMaxFrames = 65536;

// 6 statistics per frame (sup, smooth, ecc, max, min, threshold): 1.5 MiB.
// Every GPU that loads the library holds this array until the process exits.
static __device__ __align__(256) float g_af_noalloc_scratch[6 * kNoAllocMaxFrames];

namespace {

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
float *g_noalloc_ptr[kMaxDevices] = {nullptr};

// Device address of the static scratch on the current device.  In host code
// the array's name is only a host-side stand-in, so the address is looked up
// once per device (with that device current) and cached.
int noalloc_scratch(float **out)
{
    int dev = 0;
    CTBB_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) {
        set_error("adaptive filter (no allocation): device %d beyond %d", dev, kMaxDevices);
        return CTBB_ERR_ARGUMENT;
    }
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        CTBB_CUDA_TRY(cudaGetSymbolAddress(&p, g_af_noalloc_scratch));
        g_noalloc_ptr[dev] = static_cast<float *>(p);
    }
    *out = g_noalloc_ptr[dev];
    return CTBB_OK;
}

}  // namespace
}  // namespace ctbb

extern "C" int ctbb_adaptive_filter_device_noalloc(const struct recon_metadata *mr, const float *d_in,
                                                   float *d_out)
{
    using namespace ctbb;
    clear_error();
    if (!mr || !d_in || !d_out) {
        set_error("ctbb_adaptive_filter_device_noalloc: null argument");
        return CTBB_ERR_ARGUMENT;
    }
    if (mr->ri.n_proj_pull == 0 || mr->cg.n_channels == 0 || mr->cg.n_rows_raw == 0) {
        set_error("ctbb_adaptive_filter_device_noalloc: recon_metadata is not planned");
        return CTBB_ERR_STATE;
    }
    if (mr->ri.n_proj_pull > kNoAllocMaxFrames) {
        set_error("ctbb_adaptive_filter_device_noalloc: pull window of %zu frames exceeds the "
                  "fixed scratch of %zu frames; use ctbb_adaptive_filter_device",
                  mr->ri.n_proj_pull, kNoAllocMaxFrames);
        return CTBB_ERR_ARGUMENT;
    }
    CTBB_TRY(require_device());
    float *scratch = nullptr;
    CTBB_TRY(noalloc_scratch(&scratch));
    // Every statistic is written for all frames before it is read, so the
    // previous call's contents need no clearing.
    return run_adaptive_filter_with(*mr, d_in, d_out, scratch);
}
