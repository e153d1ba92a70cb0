// backproject_box.cuh -- the staged backprojector's tiles, and the detector box
// and slice classes of a visit: what backproject_staged.cu copies and how it
// reads it, computable on the host as well.
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "backproject.h"
#include "backproject_device.cuh"

namespace ctbb {

namespace {

constexpr int kGroups = 4;          // slice groups of 8: the block's 32 slices; visits of a step
constexpr int kTileY = 8;           // voxel columns of a tile along y
constexpr int kBoxRows = 8;         // detector rows of a TMA copy
constexpr float kBoxMargin = 0.05f; // rows / channels added around the box's bounds
// class of a visit for a slice group
enum : uint32_t { kSkip = 0, kFlat = 1, kInner = 2, kOther = 3, kBorder = 4, kOff = 5 };

constexpr int tile_x(int cw) { return cw == 4 ? 16 : 8; }

// Box of view t for the tile's columns x in xm +- hx, y in ym +- hy and the
// block's slices, by interval arithmetic on p, the source distance and the ray
// position: its first channel, first row | TMA copies << 16, and the class of
// each slice group (3 bits each); false when no slice of a column
// lies inside |q| < 1.
template <class Params>
__host__ __device__ __forceinline__ bool visit_box(const Params &p, float4 t, bool last, float zbase, float xm, float hx,
                                          float ym, float hy, uint32_t *chan, uint32_t *rows,
                                          uint32_t *cls)
{
    const float s = t.y, c = t.z;
    const float pc = xm * s - ym * c, ph = hx * fabsf(s) + hy * fabsf(c);
    const float tc = xm * c + ym * s, th = hx * fabsf(c) + hy * fabsf(s);
    const float p_lo = pc - ph, p_hi = pc + ph;
    const float far = fmaxf(fabsf(p_lo), fabsf(p_hi));
    const float near = (p_lo <= 0.0f && p_hi >= 0.0f) ? 0.0f : fminf(fabsf(p_lo), fabsf(p_hi));
    const float d_lo = (sqrtf(fmaxf(p.rf2 - far * far, 0.0f)) - tc - th) * p.tan_cone;
    const float d_hi = (sqrtf(fmaxf(p.rf2 - near * near, 0.0f)) - tc + th) * p.tan_cone;
    const float r1 = asinf(p_lo * p.inv_rf) * p.zrot_over_2pi, r2 = asinf(p_hi * p.inv_rf) * p.zrot_over_2pi;
    const float n_lo = zbase - t.w + fminf(r1, r2), n_hi = zbase - t.w + fmaxf(r1, r2);
    auto q_low = [&](float z) { return (n_lo + z) / (n_lo + z < 0.0f ? d_lo : d_hi); };
    auto q_high = [&](float z) { return (n_hi + z) / (n_hi + z > 0.0f ? d_lo : d_hi); };
    // up to the end of the last slice group: a warp reads for all its 8 slices,
    // also those past the block's end
    const int n_read = (p.n_slices + kSub - 1) / kSub * kSub;
    const float q_lo = q_low(0.0f), q_hi = q_high((float)(n_read - 1) * p.coll);
    if (q_lo > 1.001f || q_hi < -1.001f) return false;
    const int r_top = p.n_rows - 2;
    const int row0 = min(max((int)floorf(fmaf(q_lo, p.half_rows, p.half_rows) - kBoxMargin), 0), r_top);
    const int row1 = min(max((int)floorf(fmaf(q_hi, p.half_rows, p.half_rows) + kBoxMargin), 0), r_top) + 1;
    const float i_lo = fmaf(p_lo, p.inv_ds_half, p.two_cc) - kBoxMargin;
    const float i_hi = fmaf(p_hi, p.inv_ds_half, p.two_cc) + kBoxMargin;
    const int c_top = p.nos - 2;
    const int ch0 = min(max((int)floorf(i_lo), 0), c_top) & ~3;  // TMA copies start on 16 bytes
    // every column off the detector: nothing is read, only the weights count
    const bool off = i_hi < -1.0f || i_lo > (float)(p.nos - 1);
    *chan = (uint32_t)ch0;
    *rows = (uint32_t)row0 | (off ? 0u : (uint32_t)((row1 - row0 + kBoxRows) / kBoxRows) << 16);
    // Classes as the column form's warps take them, here for the tile's whole
    // range of q: flat (every |q| <= Q, W = 1), inner (every row inside the
    // view, in the last half turn also well below its border), border (last
    // half turn, a row at its border), other; kClassMargin covers the bounds'
    // rounding.
    constexpr float kClassMargin = 1e-5f;
    uint32_t bits = 0;
    for (int g = 0; g < kGroups; ++g) {
        const float ga = q_low((float)(g * kSub) * p.coll), gb = q_high((float)(g * kSub + kSub - 1) * p.coll);
        const float a_max = fmaxf(fabsf(ga), fabsf(gb)) + kClassMargin;
        uint32_t k = kOther;
        if (ga > 1.0f + kClassMargin || gb < -1.0f - kClassMargin || g * kSub >= p.n_slices) k = kSkip;
        else if (off) k = kOff;
        else if (p.flat_path && a_max <= kQ) k = kFlat;
        else if (a_max < kInnerMax &&
                 (!last || fmaf(a_max, p.half_rows, p.half_rows) < (float)(p.n_rows - 2) - kRowMargin))
            k = kInner;
        else if (last && fmaf(gb, p.half_rows, p.half_rows) > (float)(p.n_rows - 2) - 2.0f * kBorderBand) k = kBorder;
        bits |= k << (3 * g);
    }
    *cls = bits;
    return true;
}

}  // namespace

}  // namespace ctbb
