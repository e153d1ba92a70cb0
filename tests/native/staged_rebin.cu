// Host check of the staged rebinning's boxes: every (side, tile, chunk of
// views, channel, view) of a planned block against the box the kernel would
// copy, with the view coordinate in both forms.
#include <cmath>
#include <cstdint>

#include "rebin.h"

using namespace ctbb;

namespace {

void taps_float(int n_ffs, int proj, float ta, float off, int q, int n, int *i0, int *i1)
{
    float a = ((float)(n_ffs * proj) - ta) - off;
    if (q) a -= (float)q;
    a = n_ffs == 1 ? a : a * (n_ffs == 2 ? 0.5f : 0.25f);
    if (a > (float)(n - 1)) a = (float)n - 1.0f;
    if (a < 0.0f) a = 0.0f;
    const float fl = std::floor(a);
    *i0 = fl == fl ? (int)fl : 0;  // the device's conversion takes a NaN to 0
    *i1 = a == (float)n - 1.0f ? *i0 : *i0 + 1;
}

void taps_exact(int n_ffs, int proj, float ta, float off, int q, int n, int *i0, int *i1)
{
    const double a = ((double)n_ffs * proj - ta - off - q) / n_ffs;
    const double fl = std::floor(std::fmin(std::fmax(a, 0.0), n - 1.0));
    *i0 = fl == fl ? (int)fl : 0;
    *i1 = *i0 + 1 < n ? *i0 + 1 : n - 1;
}

}  // namespace

// Frames of the box (0: the staged kernel is not taken) in *frames, taps
// outside their box in *outside.
extern "C" int check_staged_rebin(const struct recon_metadata *mr, int *frames, long long *outside)
{
    RebinTables t;
    const int st = build_rebin_tables(*mr, &t);
    if (st) return st;
    const bool two = t.mode == RebinMode::kPhiFfs || t.mode == RebinMode::kBothFfs;
    int channels = 0;
    alignas(16) static const float raw[4] = {};
    *outside = 0;
    *frames = staged_frames(t, raw, two ? 2 : 1, &channels);
    if (!*frames) return CTBB_OK;
    const int n_tiles = (t.n_os + kRebinTile - 1) / kRebinTile, sides = (int)t.tiles.size() / n_tiles;
    for (int s = 0; s < sides; ++s)
        for (int b = 0; b < n_tiles; ++b) {
            const RebinTile &tile = t.tiles[(size_t)s * n_tiles + b];
            const int q0 = two ? 2 * s : s;
            for (int v0 = 0; v0 < t.n_views; v0 += kStagedViews)
                for (int c = b * kRebinTile; c < (b + 1) * kRebinTile && c < t.n_os; ++c) {
                    const AxisTap &tap = t.out_taps[(size_t)s * t.n_os + c];
                    for (const int i : {tap.i0, tap.i1}) {
                        const int e = two ? i & 1 : 0, ch = two ? i >> 1 : i;
                        const float ta = two ? t.focal[(size_t)(q0 + e) * t.n_channels + ch].t_alpha
                                             : t.focal[(size_t)s * t.n_os + c].t_alpha;
                        const float off = t.n_ffs == 1 ? 0.0f : t.focal_offset[q0 + e];
                        const int f0 = rebin_box_first(tile.t_max[e], off, q0 + e, t.n_ffs, v0 + t.add_projections,
                                                       t.n_proj);
                        if (ch < tile.ch0 || ch >= tile.ch0 + channels) ++*outside;
                        for (int v = v0; v < v0 + kStagedViews && v < t.n_views; ++v)
                            for (const auto taps : {taps_float, taps_exact}) {
                                int i0, i1;
                                taps(t.n_ffs, v + t.add_projections, ta, off, q0 + e, t.n_proj, &i0, &i1);
                                if (i0 < f0 || i1 >= f0 + *frames) ++*outside;
                            }
                    }
                }
        }
    return CTBB_OK;
}
