// rebin.h -- host tables and launcher of the FFS / fan-to-parallel rebinning.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "ctbb_internal.h"

namespace ctbb {

enum class RebinMode { kNoFfs, kPhiFfs, kZFfs, kBothFfs };

// interp3 taps along one axis (base, aliased upper tap, weight, 1 - weight).
struct AxisTap {
    int i0, i1;
    float u, one_minus_u;
};

// View-axis term of one (focal spot, channel): beta * n_proj_ffs / (2 pi).
struct FocalTerm {
    float t_alpha;
};

// What a tile of kRebinTile output channels of one side reads: its first raw
// channel, the channels from there, and the extremes of t_alpha over them for
// each of the side's focal spots (one or two).
constexpr int kRebinTile = 64;
struct RebinTile {
    int ch0, n_ch;
    float t_min[2], t_max[2];
};

struct RebinTables {
    RebinMode mode = RebinMode::kNoFfs;
    int n_ffs = 1, n_channels = 0, n_os = 0, n_rows_raw = 0, n_rows = 0;
    int n_proj = 0, add_projections = 0, n_views = 0, reverse_rows = 0;
    // View-axis coordinate in split form (integer frames + a fraction) instead
    // of the reference's float expression: for a window far longer than one
    // block's (the whole-scan union), where that float rounds at the
    // window's large frame offsets (rebin.cu, view_taps_split).
    int split_view_coord = 0;
    std::vector<AxisTap> out_taps;   // [side][n_os]
    std::vector<FocalTerm> focal;    // no/z-FFS: [side][n_os]; phi/both: [focal][n_channels]
    std::vector<RebinTile> tiles;    // [side][tiles of the output channels]
    std::vector<float> focal_offset; // d_alpha_r * n_proj_ffs / (2 pi) per focal spot
};

struct CopyError;  // tma.cuh: a context's word for copies that did not arrive

struct DeviceRebinTables {
    void *base = nullptr;
    size_t capacity = 0;
    AxisTap *taps = nullptr;
    FocalTerm *focal = nullptr;
    RebinTile *tiles = nullptr;
};

int build_rebin_tables(const struct recon_metadata &mr, RebinTables *t);

// The staged kernel (rebin.cu): a CTA's views of one side, and the first frame
// of its box of focal spot q (offset off, largest t_alpha t_max): one before
// the lowest view coordinate (whose float rounding is far below a frame),
// inside the scan as the taps are.
constexpr int kStagedViews = 16;
__host__ __device__ inline int rebin_box_first(float t_max, float off, int q, int n_ffs, int proj, int n_proj)
{
    const float c = t_max + off + (float)q;
    const int lowest = proj - (int)ceilf(c / (float)n_ffs) - 1;
    return lowest < 0 ? 0 : (lowest > n_proj - 1 ? n_proj - 1 : lowest);
}
// Frames of the staged kernel's boxes, or 0 where it does not apply: rows off
// 16-byte boundaries, a tile wider than the box, t_alpha moving so fast that
// two boxes do not fit beside another CTA's (few, wide channels), or a channel
// whose t_alpha is not finite (past 90 degrees): the gathering kernel clamps
// its view to the scan, but no box can be placed around it.
int staged_frames(const RebinTables &t, const float *d_raw, int spots, int *channels);

int upload_rebin_tables(const RebinTables &t, DeviceRebinTables *dt, cudaStream_t stream);
// Views [v_begin, v_end) of the output (v_end < 0: all views).
int launch_rebin(const RebinTables &t, const DeviceRebinTables &dt, const float *d_raw,
                 float *d_out, CopyError &errors, cudaStream_t stream, int v_begin = 0, int v_end = -1);
// Frames of the pull window view v reads (focal-spot frames of the view-axis
// taps of every channel): all lie below rebin_frames_needed(t, v).
int rebin_frames_needed(const RebinTables &t, int v);

}  // namespace ctbb
