// rebin.cu -- flying-focal-spot split + fan-to-parallel rebinning.
//
// One fused kernel per FFS mode replaces the reference's reshape /
// azimuthal / radial kernel chain (src/rebin_filter.cu:58-912) and the CPU twin
// it must match (src/rebin_filter_cpu.cu:95-645):
//
//   * no FFS  (rebin_nffs_cpu :95-159) and z-FFS (rebin_zffs_cpu :290-416):
//     one bilinear sample in (channel, view) per output sample;
//   * phi-FFS (rebin_pffs_cpu :161-288) and phi+z-FFS (rebin_affs_cpu :418-645):
//     the reference first rebins azimuthally into an oversampled intermediate
//     (channels 2ch / 2ch+1 from the +da / -da focal spots) and then radially
//     along that intermediate's channel axis.  Here each output sample evaluates
//     the two intermediate samples it needs on the fly, so the intermediate is
//     never stored.
//
// Geometry-only quantities (fan angles, beta_lookup search, view offsets) are
// computed on the host with the reference's float expressions; the kernels do
// clamps, floors, multiplies and adds only, written with __f*_rn intrinsics so
// that no multiply-add is fused.  The unfiltered result is therefore bit-exact
// with the reference CPU path compiled without FMA contraction.
//
// Two forms with the same taps and arithmetic.  The staged one copies the
// frames that a tile of output channels and views can read to shared memory by
// TMA; the gathering one (channel counts that are not a multiple of 4, raw
// pointers off 16 bytes, tiles too wide for the box) reads them through L1.  In
// both a thread covers one output channel and 4 raw rows, so the view-axis taps
// of a (channel, view) are computed once for its rows.  A launch may cover a
// range of views (the streamed whole-scan path).
//
// Output layout: rebin[view][out_row][channel_os], views = n_proj/n_ffs -
// 2*add_projections (the leading add_projections views are dropped, as the
// reference's copy loops do, e.g. src/rebin_filter_cpu.cu:119-131).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "ctbb_internal.h"
#include "cuda_util.cuh"
#include "rebin.h"
#include "tma.cuh"

namespace ctbb {

namespace {

// ---- host restatements of the reference's float geometry helpers ----------
// src/rebin_filter_cpu.cu:37-65.  C++ overloads as in the reference: pow(2.0f,
// int) promotes to double, so b0 is computed in double and rounded to float.

float angle_f(float x1, float x2, float y1, float y2)
{
    return std::asin((x1 * y2 - x2 * y1) / (std::sqrt(x1 * x1 + x2 * x2) * std::sqrt(y1 * y1 + y2 * y2)));
}

float beta_rk_f(float da, float dr, float channel, int os_flag, const struct ct_geom &cg)
{
    float b0 = (float)((channel - std::pow(2.0f, os_flag) * cg.central_channel) *
                       (cg.fan_angle_increment / std::pow(2.0f, os_flag)));
    return angle_f(-(cg.r_f + dr), -(da), -(cg.src_to_det * std::cos(b0) + dr),
                   -(cg.src_to_det * std::sin(b0) + da));
}

float d_alpha_r_f(float da, float dr, const struct ct_geom &cg)
{
    return angle_f(cg.r_f, 0, cg.r_f + dr, da);
}

float r_fr_f(float da, float dr, const struct ct_geom &cg)
{
    return std::sqrt((cg.r_f + dr) * (cg.r_f + dr) + da * da);
}

// get_beta_idx with the search begun where the last one ended: every entry
// before it is below the last beta, so for a beta no smaller the first entry
// that is not below it is the same as from 0 (1472 searches of 1472 entries
// took the host 1.1 ms of every rebin call).
struct BetaSearch {
    const float *lookup;
    int n, from = 0;
    float last = -INFINITY;
};

float get_beta_idx_f(float beta, BetaSearch &b)
{
    const float *lookup = b.lookup;
    const int n = b.n;
    int lo = beta >= b.last ? b.from : 0;
    while (beta > lookup[lo] && lo < (n - 1)) lo++;
    b.from = lo;
    b.last = beta;
    if (lo == 0) lo++;
    return (float)lo - 1.0f + (beta - lookup[lo - 1]) / (lookup[lo] - lookup[lo - 1]);
}

// Clamp + floor + alias rule of interp3 (src/interp.cu:66-130) along one axis
// whose coordinate does not depend on the view: base tap, upper tap and
// weight, evaluated exactly as interp3 does.
void axis_taps(float idx, int dim, int *i0, int *i1, float *u, float *one_minus_u)
{
    if (idx > (float)(dim - 1)) idx = (float)dim - 1.0f;
    if (idx < 0) idx = 0.0f;
    float fl = std::floor(idx);
    *u = idx - fl;
    *one_minus_u = 1.0f - *u;
    *i0 = fl == fl ? (int)fl : 0;  // a channel past 90 degrees: weights that are not numbers, taps in range
    *i1 = (idx == (float)dim - 1.0f) ? *i0 : *i0 + 1;
}

}  // namespace

// --------------------------------------------------------------------------
// Host tables
// --------------------------------------------------------------------------

int build_rebin_tables(const struct recon_metadata &mr, RebinTables *t)
{
    const struct ct_geom &cg = mr.cg;
    const struct recon_params &rp = mr.rp;
    const int N = (int)cg.n_channels, Nos = (int)cg.n_channels_oversampled;
    const float pi = kPiRebin;
    const float two_pi = 2.0f * pi;
    t->n_ffs = (int)mr.ri.n_ffs;
    t->n_channels = N;
    t->n_os = Nos;
    t->n_rows_raw = (int)cg.n_rows_raw;
    t->n_rows = (int)cg.n_rows;
    t->n_proj = (int)(mr.ri.n_proj_pull / mr.ri.n_ffs);
    t->add_projections = (int)cg.add_projections;
    t->n_views = t->n_proj - 2 * t->add_projections;
    t->reverse_rows = cg.reverse_row_interleave ? 1 : 0;
    if (t->n_views <= 0) {
        set_error("rebin: pull window of %zu frames keeps no views", mr.ri.n_proj_pull);
        return CTBB_ERR_STATE;
    }
    t->out_taps.assign(2 * (size_t)Nos, AxisTap{});
    t->focal.assign(4 * (size_t)N, FocalTerm{});
    t->focal_offset.assign(4, 0.0f);

    auto set_tap = [&](int s, int c, float bidx, int dim) {
        AxisTap &a = t->out_taps[(size_t)s * Nos + c];
        axis_taps(bidx, dim, &a.i0, &a.i1, &a.u, &a.one_minus_u);
    };

    if (t->n_ffs == 1) {
        // rebin_nffs_cpu :107-117
        t->mode = RebinMode::kNoFfs;
        t->focal.assign((size_t)Nos, FocalTerm{});
        for (int c = 0; c < Nos; ++c) {
            const float beta = std::asin(((float)c - 2 * cg.central_channel) * (cg.fan_angle_increment / 2));
            float beta_idx = beta / cg.fan_angle_increment + cg.central_channel;
            set_tap(0, c, beta_idx, N);
            t->focal[c].t_alpha = beta * (float)cg.n_proj_turn / (2.0f * pi);
        }
    } else if (t->n_ffs == 2 && rp.z_ffs == 1) {
        // rebin_zffs_cpu :297-352
        t->mode = RebinMode::kZFfs;
        const double da = 0.0;
        const double dr = cg.src_to_det * rp.coll_slicewidth /
                          (4.0 * (cg.src_to_det - cg.r_f) * std::tan(cg.anode_angle));
        std::vector<float> lk1(N), lk2(N);
        for (int i = 0; i < N; i++) {
            lk1[i] = beta_rk_f((float)da, (float)-dr, (float)i, 0, cg);
            lk2[i] = beta_rk_f((float)da, (float)dr, (float)i, 0, cg);
        }
        t->focal.assign(2 * (size_t)Nos, FocalTerm{});
        BetaSearch at1{lk1.data(), N}, at2{lk2.data(), N};
        float dal1 = d_alpha_r_f((float)da, (float)-dr, cg) * (float)cg.n_proj_ffs / (2.0f * pi);
        float dal2 = d_alpha_r_f((float)da, (float)dr, cg) * (float)cg.n_proj_ffs / (2.0f * pi);
        t->focal_offset[0] = dal1;
        t->focal_offset[1] = dal2;
        for (int c = 0; c < Nos; ++c) {
            float b1 = std::asin(((float)c - 2.0f * cg.central_channel) * (cg.fan_angle_increment / 2.0f) *
                                 cg.r_f / r_fr_f(0.0f, (float)-dr, cg));
            float b2 = std::asin(((float)c - 2.0f * cg.central_channel) * (cg.fan_angle_increment / 2.0f) *
                                 cg.r_f / r_fr_f(0.0f, (float)dr, cg));
            set_tap(0, c, get_beta_idx_f(b1, at1), N);
            set_tap(1, c, get_beta_idx_f(b2, at2), N);
            t->focal[c].t_alpha = b1 * (float)cg.n_proj_ffs / (2.0f * pi);
            t->focal[(size_t)Nos + c].t_alpha = b2 * (float)cg.n_proj_ffs / (2.0f * pi);
        }
    } else if (t->n_ffs == 2) {
        // rebin_pffs_cpu :165-246
        t->mode = RebinMode::kPhiFfs;
        const double da = cg.src_to_det * cg.r_f * cg.fan_angle_increment /
                          (4.0f * (cg.src_to_det - cg.r_f));
        std::vector<float> lookup(Nos);
        float dal_p = d_alpha_r_f((float)da, 0, cg) * (float)cg.n_proj_ffs / (2.0f * pi);
        float dal_m = d_alpha_r_f((float)-da, 0, cg) * (float)cg.n_proj_ffs / (2.0f * pi);
        t->focal_offset[0] = dal_p;
        t->focal_offset[1] = dal_m;
        for (int ch = 0; ch < N; ++ch) {
            float b1 = beta_rk_f((float)da, 0, (float)ch, 0, cg);
            float b2 = beta_rk_f((float)-da, 0, (float)ch, 0, cg);
            lookup[2 * ch] = b1;
            lookup[2 * ch + 1] = b2;
            t->focal[0 * (size_t)N + ch].t_alpha = b1 * (float)cg.n_proj_ffs / (2.0f * pi);
            t->focal[1 * (size_t)N + ch].t_alpha = b2 * (float)cg.n_proj_ffs / (2.0f * pi);
        }
        BetaSearch at{lookup.data(), Nos};
        for (int c = 0; c < Nos; ++c) {
            float beta = std::asin((c - 2 * cg.central_channel) * (cg.fan_angle_increment / 2));
            set_tap(0, c, get_beta_idx_f(beta, at), Nos);
        }
    } else if (t->n_ffs == 4) {
        // rebin_affs_cpu :424-601
        t->mode = RebinMode::kBothFfs;
        const double da = cg.src_to_det * cg.r_f * cg.fan_angle_increment /
                          (4.0f * (cg.src_to_det - cg.r_f));
        const double dr = cg.src_to_det * rp.coll_slicewidth /
                          (4.0 * (cg.src_to_det - cg.r_f) * std::tan(cg.anode_angle));
        std::vector<float> lk1(Nos), lk2(Nos);
        // focal order within a group of 4 frames: (+da,-dr) (-da,-dr) (+da,+dr) (-da,+dr)
        const float sda[4] = {(float)da, (float)-da, (float)da, (float)-da};
        const float sdr[4] = {(float)-dr, (float)-dr, (float)dr, (float)dr};
        for (int q = 0; q < 4; ++q)
            t->focal_offset[q] = d_alpha_r_f(sda[q], sdr[q], cg) * (float)cg.n_proj_ffs / (2.0f * pi);
        for (int ch = 0; ch < N; ++ch) {
            for (int q = 0; q < 4; ++q) {
                float b = beta_rk_f(sda[q], sdr[q], (float)ch, 0, cg);
                t->focal[(size_t)q * N + ch].t_alpha = b * (float)cg.n_proj_ffs / (2.0f * pi);
                if (q < 2) lk1[2 * ch + q] = b;
                else lk2[2 * ch + (q - 2)] = b;
            }
        }
        BetaSearch at1{lk1.data(), Nos}, at2{lk2.data(), Nos};
        for (int c = 0; c < Nos; ++c) {
            float b1 = std::asin((c - 2 * cg.central_channel) * (cg.fan_angle_increment / 2) * cg.r_f /
                                 r_fr_f(0.0f, (float)-dr, cg));
            float b2 = std::asin((c - 2 * cg.central_channel) * (cg.fan_angle_increment / 2) * cg.r_f /
                                 r_fr_f(0.0f, (float)dr, cg));
            set_tap(0, c, get_beta_idx_f(b1, at1), Nos);
            set_tap(1, c, get_beta_idx_f(b2, at2), Nos);
        }
    } else {
        set_error("rebin: unsupported n_ffs %d", t->n_ffs);
        return CTBB_ERR_CONFIG;
    }
    (void)two_pi;
    // the tiles' reads, from the taps and terms above
    const bool two_stage = t->mode == RebinMode::kPhiFfs || t->mode == RebinMode::kBothFfs;
    const int sides = two_stage ? (t->n_ffs == 4 ? 2 : 1) : t->n_ffs;
    const int n_tiles = (Nos + kRebinTile - 1) / kRebinTile;
    t->tiles.assign((size_t)sides * n_tiles, RebinTile{});
    for (int s = 0; s < sides; ++s)
        for (int b = 0; b < n_tiles; ++b) {
            RebinTile &tile = t->tiles[(size_t)s * n_tiles + b];
            int lo = N, hi = 0;
            for (int e = 0; e < 2; ++e) {
                tile.t_min[e] = INFINITY;
                tile.t_max[e] = -INFINITY;
            }
            auto reads = [&](int ch, int e, float t_alpha) {
                lo = std::min(lo, ch);
                hi = std::max(hi, ch);
                if (!std::isfinite(t_alpha + t->focal_offset[two_stage ? 2 * s + e : s])) {  // no box holds its views (see staged_frames)
                    tile.t_min[e] = -INFINITY;
                    tile.t_max[e] = INFINITY;
                }
                tile.t_min[e] = std::min(tile.t_min[e], t_alpha);
                tile.t_max[e] = std::max(tile.t_max[e], t_alpha);
            };
            for (int c = b * kRebinTile; c < std::min(Nos, (b + 1) * kRebinTile); ++c) {
                const AxisTap &tap = t->out_taps[(size_t)s * Nos + c];
                for (const int i : {tap.i0, tap.i1}) {
                    if (two_stage) reads(i >> 1, i & 1, t->focal[(size_t)(2 * s + (i & 1)) * N + (i >> 1)].t_alpha);
                    else reads(i, 0, t->focal[(size_t)s * Nos + c].t_alpha);
                }
            }
            tile.ch0 = lo & ~3;  // TMA copies start on 16 bytes
            tile.n_ch = hi - tile.ch0 + 1;
        }
    return CTBB_OK;
}

// --------------------------------------------------------------------------
// Device helpers
// --------------------------------------------------------------------------

struct RebinParams {
    const float *raw;           // [P][R_raw][N]
    float *out;                 // [V][R][Nos]
    const AxisTap *taps;        // [2][Nos]
    const FocalTerm *focal;     // mode dependent
    float focal_offset[4];
    int n_ffs, N, Nos, R_raw, R, n_proj, add, n_views, reverse_rows;
    int split_view_coord;
    int v_begin, v_end;  // views this launch writes
};

// View-axis coordinate of focal spot q at view proj, divided down to the index
// of that focal spot's own frame sequence (src/rebin_filter_cpu.cu:210-219, :346-356,
// :519-544): ((n_ffs*proj - t_alpha) - t_offset - q) / n_ffs.
__device__ __forceinline__ float focal_alpha(int n_ffs, int proj, float t_alpha, float t_off, int q)
{
    float a = __fsub_rn(__fsub_rn((float)(n_ffs * proj), t_alpha), t_off);
    if (q) a = __fsub_rn(a, (float)q);
    return n_ffs == 1 ? a : __fmul_rn(a, n_ffs == 2 ? 0.5f : 0.25f);
}

// interp3 taps along the view axis (clamp to [0, n-1], alias at the edge).
__device__ __forceinline__ void view_taps(float a, int n, int *i0, int *i1, float *w)
{
    if (a > (float)(n - 1)) a = (float)n - 1.0f;
    if (a < 0.0f) a = 0.0f;
    float fl = floorf(a);
    *w = __fsub_rn(a, fl);
    *i0 = (int)fl;
    *i1 = (a == (float)n - 1.0f) ? *i0 : *i0 + 1;
}

// The same taps from the coordinate ((n_ffs proj - t_alpha) - t_off - q) /
// n_ffs evaluated in split form.  In float that expression rounds at the
// magnitude of n_ffs proj: within one block's pull window (proj below ~2500)
// to 5e-4 frames, but in the whole-scan union (proj up to ~11000 at 40
// turns) to 4e-3 frames, which moves the view weights of the later blocks by
// up to 1e-3.  Here c = t_alpha + t_off + q (a few hundred frames) is split
// into floor(c) and the exact remainder c - floor(c); n_ffs proj - floor(c)
// is an exact integer J = n_ffs Q + m with 0 <= m < n_ffs, and the coordinate
// is Q + (m - (c - floor(c))) / n_ffs, whose fraction is rounded at a
// magnitude below n_ffs.  The result differs from the exact coordinate by
// about 1e-7 views, from any block's own float coordinate by at most that
// block's rounding.  Same clamp and edge alias as view_taps.
__device__ __forceinline__ void view_taps_split(int n_ffs, int proj, float t_alpha, float t_off, int q, int n,
                                                int *i0, int *i1, float *w)
{
    float c = __fadd_rn(__fadd_rn(t_alpha, t_off), (float)q);
    float cf = floorf(c);
    float c_frac = __fsub_rn(c, cf);  // exact: same binade or finer
    int J = n_ffs * proj - (int)cf;
    // floor(J / n_ffs) and its remainder, n_ffs a power of two (1, 2, 4): an
    // arithmetic shift floors for negative J as well
    const int lg = n_ffs >> 1;  // log2 n_ffs for 1, 2, 4
    int Q = J >> lg;
    int m = J - (Q << lg);
    float r = __fsub_rn((float)m, c_frac);  // in (-1, n_ffs)
    r = n_ffs == 1 ? r : __fmul_rn(r, n_ffs == 2 ? 0.5f : 0.25f);
    if (r < 0.0f) {  // floor
        Q -= 1;
        r = __fadd_rn(r, 1.0f);
        if (r >= 1.0f) {  // -r rounded to below 1 ulp of 1
            Q += 1;
            r = 0.0f;
        }
    }
    if (Q < 0) {
        *i0 = 0;
        *i1 = n > 1 ? 1 : 0;
        *w = 0.0f;
    } else if (Q > n - 1 || (Q == n - 1 && r > 0.0f)) {
        *i0 = n - 1;
        *i1 = n - 1;
        *w = 0.0f;
    } else {
        *i0 = Q;
        *i1 = (Q == n - 1) ? Q : Q + 1;
        *w = r;
    }
}

// Views per thread: the per-channel taps and focal terms are loaded once and
// reused along the view axis.
constexpr int kViewsPerThread = 8;

// --------------------------------------------------------------------------
// Kernels.  Idx is the index type of the raw and output arrays (32-bit when
// both hold fewer than 2^31 samples).
// --------------------------------------------------------------------------

// Raw rows per thread: the view-axis taps of a (channel, view) are computed
// once and used for every row of the group.  Measured on a config-2 window
// (phi+z FFS): 1 row 717 us, 2 rows 730, 4 rows 572, 8 rows 645, 16 rows
// 1003 (the L2 stops holding the rows in flight: 4.3 GB of reads for 1.1 GB).
constexpr int kRowsPerThread = 4;

// no-FFS and z-FFS: bilinear in (channel, view).  grid: x channel blocks,
// y groups of kRowsPerThread raw rows, z chunks of kViewsPerThread views.
template <class Idx>
__global__ void rebin_bilinear_kernel(RebinParams p)
{
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    int r0 = blockIdx.y * kRowsPerThread;
    int r1 = min(r0 + kRowsPerThread, p.R_raw);
    int v0 = p.v_begin + blockIdx.z * kViewsPerThread;
    if (c >= p.Nos) return;
    const Idx frame_stride = (Idx)p.R_raw * p.N;
    const Idx nos = (Idx)p.Nos;
    for (int s = 0; s < p.n_ffs; ++s) {
        const AxisTap tap = p.taps[s * p.Nos + c];
        const float t_alpha = p.focal[s * p.Nos + c].t_alpha;
        const float t_off = p.n_ffs == 1 ? 0.0f : p.focal_offset[s];
        const float omu = tap.one_minus_u, u = tap.u;
        const float *base = p.raw + s * frame_stride;
        for (int v = v0; v < min(v0 + kViewsPerThread, p.v_end); ++v) {
            int i0, i1;
            float w;
            if (p.split_view_coord)
                view_taps_split(p.n_ffs, v + p.add, t_alpha, t_off, s, p.n_proj, &i0, &i1, &w);
            else
                view_taps(focal_alpha(p.n_ffs, v + p.add, t_alpha, t_off, s), p.n_proj, &i0, &i1, &w);
            const float *f0 = base + (Idx)(p.n_ffs * i0) * frame_stride;
            const float *f1 = base + (Idx)(p.n_ffs * i1) * frame_stride;
            float omw = __fsub_rn(1.0f, w);
            float *out_v = p.out + (Idx)v * p.R * nos + c;
#pragma unroll 4
            for (int row = r0; row < r1; ++row) {
                const Idx ro = (Idx)row * p.N;
                float a1 = __ldg(f0 + ro + tap.i0), a2 = __ldg(f0 + ro + tap.i1);
                float a5 = __ldg(f1 + ro + tap.i0), a6 = __ldg(f1 + ro + tap.i1);
                float t1 = __fmul_rn(__fmul_rn(a1, omu), omw);
                float t2 = __fmul_rn(__fmul_rn(a2, u), omw);
                float t5 = __fmul_rn(__fmul_rn(a5, omu), w);
                float t6 = __fmul_rn(__fmul_rn(a6, u), w);
                int out_row = row;
                if (p.n_ffs == 2) out_row = 2 * row + (p.reverse_rows ? 1 - s : s);
                out_v[(Idx)out_row * nos] = __fadd_rn(__fadd_rn(__fadd_rn(t1, t2), t5), t6);
            }
        }
    }
}

// phi-FFS and phi+z-FFS: radial interpolation between two samples of the
// (virtual) azimuthally rebinned intermediate, each a view-axis lerp of one
// focal spot.  For phi+z-FFS side s = 0 (-dr) uses focal spots 0/1 and s = 1
// (+dr) focal spots 2/3.
template <class Idx>
__global__ void rebin_two_stage_kernel(RebinParams p)
{
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    int r0 = blockIdx.y * kRowsPerThread;
    int r1 = min(r0 + kRowsPerThread, p.R_raw);
    int v0 = p.v_begin + blockIdx.z * kViewsPerThread;
    if (c >= p.Nos) return;
    const Idx frame_stride = (Idx)p.R_raw * p.N;
    const Idx nos = (Idx)p.Nos;
    int sides = p.n_ffs == 4 ? 2 : 1;
    for (int s = 0; s < sides; ++s) {
        const AxisTap tap = p.taps[s * p.Nos + c];
        int qb = 2 * s;
        int q0 = qb + (tap.i0 & 1), ch0 = tap.i0 >> 1;
        int q1 = qb + (tap.i1 & 1), ch1 = tap.i1 >> 1;
        const float ta0 = p.focal[q0 * p.N + ch0].t_alpha, to0 = p.focal_offset[q0];
        const float ta1 = p.focal[q1 * p.N + ch1].t_alpha, to1 = p.focal_offset[q1];
        const float *b0 = p.raw + ch0 + q0 * frame_stride;
        const float *b1 = p.raw + ch1 + q1 * frame_stride;
        for (int v = v0; v < min(v0 + kViewsPerThread, p.v_end); ++v) {
            int proj = v + p.add;
            int i0, i1, j0, j1;
            float w0, w1;
            if (p.split_view_coord) {
                view_taps_split(p.n_ffs, proj, ta0, to0, q0, p.n_proj, &i0, &i1, &w0);
                view_taps_split(p.n_ffs, proj, ta1, to1, q1, p.n_proj, &j0, &j1, &w1);
            } else {
                view_taps(focal_alpha(p.n_ffs, proj, ta0, to0, q0), p.n_proj, &i0, &i1, &w0);
                view_taps(focal_alpha(p.n_ffs, proj, ta1, to1, q1), p.n_proj, &j0, &j1, &w1);
            }
            const float *f00 = b0 + (Idx)(p.n_ffs * i0) * frame_stride;
            const float *f01 = b0 + (Idx)(p.n_ffs * i1) * frame_stride;
            const float *f10 = b1 + (Idx)(p.n_ffs * j0) * frame_stride;
            const float *f11 = b1 + (Idx)(p.n_ffs * j1) * frame_stride;
            const float omw0 = __fsub_rn(1.0f, w0), omw1 = __fsub_rn(1.0f, w1);
            float *out_v = p.out + (Idx)v * p.R * nos + c;
#pragma unroll 4
            for (int row = r0; row < r1; ++row) {
                const Idx ro = (Idx)row * p.N;
                float T0 = __fadd_rn(__fmul_rn(__ldg(f00 + ro), omw0), __fmul_rn(__ldg(f01 + ro), w0));
                float T1 = __fadd_rn(__fmul_rn(__ldg(f10 + ro), omw1), __fmul_rn(__ldg(f11 + ro), w1));
                int out_row = row;
                if (p.n_ffs == 4) out_row = 2 * row + (p.reverse_rows ? 1 - s : s);
                out_v[(Idx)out_row * nos] = __fadd_rn(__fmul_rn(T0, tap.one_minus_u), __fmul_rn(T1, tap.u));
            }
        }
    }
}

// ---- staged form ---------------------------------------------------------
//
// A gather of the kernels above takes 27 wavefronts of the L1 data pipe per
// warp of outputs (81 % of its peak on a config-2 window): t_alpha moves by a
// frame every few channels, so the 32 channels of a warp fall on four or five
// frames of each focal spot, and one wavefront serves one of them.  Here a CTA
// (64 output channels, kRowsPerThread raw rows, kStagedViews views of one
// side) copies the frames its views can read -- a box of channels x rows x
// frames per focal spot -- into shared memory by TMA (two copies) and gathers
// from there, where frames lie a whole number of bank rounds apart and lanes of
// consecutive channels do not collide.  Same taps, same arithmetic, same bits.
// Small tiles: t_alpha's span over a tile adds frames to every box, so 128
// channels (96 KB of boxes, 2 CTAs per SM) moved 3.2 GB from L2 and took 592
// us on a config-2 window where 64 (37 KB, 6 CTAs) move 2.55 GB and took 415
// (390 now); 32 views to a box 550, 256 threads 454; gathering 611.  What bounds
// it now is the L2 traffic of the boxes (6.6 TB/s) beside 5.2 TB/s of HBM.
constexpr int kNarrowBox = 40, kWideBox = 48;  // channels of a box: a tile's, wider with a z flying focal spot

struct StagedRebin {
    const RebinTile *tiles;
    int n_tiles, n_groups, frames;  // frames of a box
};

template <bool TWO, int CH>
__global__ void __launch_bounds__(128) rebin_staged_kernel(RebinParams p, StagedRebin g,
                                                           const __grid_constant__ CUtensorMap map, int *error)
{
    extern __shared__ __align__(128) float box[];
    constexpr int kSpots = TWO ? 2 : 1;
    constexpr int kFrame = kRowsPerThread * CH;  // floats between frames: a multiple of 32
    static_assert(kFrame % 32 == 0, "frames share their banks");
    __shared__ __align__(8) unsigned long long full;
    const int side = blockIdx.y / g.n_groups, r0 = (blockIdx.y - side * g.n_groups) * kRowsPerThread;
    const int v0 = p.v_begin + blockIdx.z * kStagedViews, v1 = min(v0 + kStagedViews, p.v_end);
    const RebinTile tile = g.tiles[side * g.n_tiles + blockIdx.x];
    const int q0 = TWO ? 2 * side : side;  // the side's first focal spot
    int f0[kSpots];  // first frame of each box
#pragma unroll
    for (int e = 0; e < kSpots; ++e) {
        const float off = p.n_ffs == 1 ? 0.0f : p.focal_offset[q0 + e];
        f0[e] = rebin_box_first(tile.t_max[e], off, q0 + e, p.n_ffs, v0 + p.add, p.n_proj);
    }
    const uint32_t bar = smem_address(&full);
    if (threadIdx.x == 0) {
        barrier_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        barrier_arrive_expect(bar, (uint32_t)(kSpots * g.frames * kFrame) * 4u);
#pragma unroll
        for (int e = 0; e < kSpots; ++e)
            asm volatile(
                "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
                "%5}], [%6];" ::"r"(smem_address(box + e * g.frames * kFrame)),
                "l"(reinterpret_cast<uint64_t>(&map)), "r"(tile.ch0), "r"(r0), "r"(q0 + e), "r"(f0[e]), "r"(bar)
                : "memory");
    }
    __syncthreads();
    const int c = blockIdx.x * kRebinTile + (threadIdx.x & (kRebinTile - 1));
    const bool in = c < p.Nos;
    // this thread's half of the views
    constexpr int kHalf = kStagedViews / 2;
    const int w0 = v0 + (int)(threadIdx.x / kRebinTile) * kHalf, w1 = min(w0 + kHalf, v1);
    const int n_rows = min(kRowsPerThread, p.R_raw - r0);
    AxisTap tap = {};
    float ta0 = 0.0f, ta1 = 0.0f, to0 = 0.0f, to1 = 0.0f;
    int e0 = 0, e1 = 0;  // focal spots of the two channel taps, within the side
    const float *b0 = box, *b1 = box;
    if (in) {
        tap = p.taps[side * p.Nos + c];
        if (TWO) {
            e0 = tap.i0 & 1;
            e1 = tap.i1 & 1;
            ta0 = p.focal[(q0 + e0) * p.N + (tap.i0 >> 1)].t_alpha;
            ta1 = p.focal[(q0 + e1) * p.N + (tap.i1 >> 1)].t_alpha;
            to0 = p.focal_offset[q0 + e0];
            to1 = p.focal_offset[q0 + e1];
            b0 = box + (e0 ? g.frames * kFrame : 0) - (e0 ? f0[kSpots - 1] : f0[0]) * kFrame + (tap.i0 >> 1) - tile.ch0;
            b1 = box + (e1 ? g.frames * kFrame : 0) - (e1 ? f0[kSpots - 1] : f0[0]) * kFrame + (tap.i1 >> 1) - tile.ch0;
        } else {
            ta0 = p.focal[side * p.Nos + c].t_alpha;
            to0 = p.n_ffs == 1 ? 0.0f : p.focal_offset[side];
            b0 = box - f0[0] * kFrame + tap.i0 - tile.ch0;
            b1 = box - f0[0] * kFrame + tap.i1 - tile.ch0;
        }
    }
    const bool copied = barrier_wait(bar, 0);
    const bool z_ffs = TWO ? p.n_ffs == 4 : p.n_ffs == 2;
    const size_t nos = (size_t)p.Nos;
    const int out_first = z_ffs ? 2 * r0 + (p.reverse_rows ? 1 - side : side) : r0;
    const size_t out_step = (z_ffs ? 2 : 1) * nos;
    if (!copied) {
        *reinterpret_cast<volatile int *>(error) = 1;
        wait_for_stray_copies();
        if (in)
            for (int v = w0; v < w1; ++v)
                for (int r = 0; r < n_rows; ++r)
                    p.out[((size_t)v * p.R + out_first) * nos + c + r * out_step] = __int_as_float(0x7fffffff);
        return;
    }
    if (!in) return;
    for (int v = w0; v < w1; ++v) {
        const int proj = v + p.add;
        int i0, i1, j0 = 0, j1 = 0;
        float wa, wb = 0.0f;
        if (p.split_view_coord) {
            view_taps_split(p.n_ffs, proj, ta0, to0, q0 + e0, p.n_proj, &i0, &i1, &wa);
            if (TWO) view_taps_split(p.n_ffs, proj, ta1, to1, q0 + e1, p.n_proj, &j0, &j1, &wb);
        } else {
            view_taps(focal_alpha(p.n_ffs, proj, ta0, to0, q0 + e0), p.n_proj, &i0, &i1, &wa);
            if (TWO) view_taps(focal_alpha(p.n_ffs, proj, ta1, to1, q0 + e1), p.n_proj, &j0, &j1, &wb);
        }
        float *out = p.out + ((size_t)v * p.R + out_first) * nos + c;
        const float oma = __fsub_rn(1.0f, wa), omb = __fsub_rn(1.0f, wb);
        const float *x00 = b0 + i0 * kFrame, *x01 = b0 + i1 * kFrame;
        const float *x10 = b1 + (TWO ? j0 : i0) * kFrame, *x11 = b1 + (TWO ? j1 : i1) * kFrame;
#pragma unroll
        for (int r = 0; r < kRowsPerThread; ++r) {
            if (r >= n_rows) break;
            const int o = r * CH;
            float y;
            if (TWO) {
                const float T0 = __fadd_rn(__fmul_rn(x00[o], oma), __fmul_rn(x01[o], wa));
                const float T1 = __fadd_rn(__fmul_rn(x10[o], omb), __fmul_rn(x11[o], wb));
                y = __fadd_rn(__fmul_rn(T0, tap.one_minus_u), __fmul_rn(T1, tap.u));
            } else {
                const float t1 = __fmul_rn(__fmul_rn(x00[o], tap.one_minus_u), oma);
                const float t2 = __fmul_rn(__fmul_rn(x10[o], tap.u), oma);
                const float t5 = __fmul_rn(__fmul_rn(x01[o], tap.one_minus_u), wa);
                const float t6 = __fmul_rn(__fmul_rn(x11[o], tap.u), wa);
                y = __fadd_rn(__fadd_rn(__fadd_rn(t1, t2), t5), t6);
            }
            out[r * out_step] = y;
        }
    }
}

int staged_frames(const RebinTables &t, const float *d_raw, int spots, int *channels)
{
    if (t.n_channels % 4 != 0 || ((uintptr_t)d_raw & 15) != 0) return 0;
    float span = 0.0f;
    int widest = 0;
    for (const RebinTile &tile : t.tiles) {
        widest = std::max(widest, tile.n_ch);
        for (int e = 0; e < spots; ++e)
            if (tile.t_max[e] >= tile.t_min[e]) span = std::max(span, tile.t_max[e] - tile.t_min[e]);
    }
    if (widest > kWideBox) return 0;
    *channels = widest <= kNarrowBox ? kNarrowBox : kWideBox;
    // the views, t_alpha's span, and a frame of margin and the upper tap at either end
    const float frames = (float)kStagedViews + std::ceil(span / (float)t.n_ffs) + 5.0f;
    return frames <= 256.0f && frames * spots * kRowsPerThread * *channels * 4 <= 110 * 1024 ? (int)frames : 0;
}

int launch_rebin_staged(const RebinTables &t, const DeviceRebinTables &dt, const RebinParams &p, bool two, int frames,
                        int channels, CopyError &errors, cudaStream_t stream)
{
    const cuuint64_t row = (cuuint64_t)t.n_channels * 4, frame = row * t.n_rows_raw;
    const cuuint64_t dims[4] = {(cuuint64_t)t.n_channels, (cuuint64_t)t.n_rows_raw, (cuuint64_t)t.n_ffs,
                                (cuuint64_t)t.n_proj};
    const cuuint64_t strides[3] = {row, frame, frame * t.n_ffs};
    const cuuint32_t box[4] = {(cuuint32_t)channels, kRowsPerThread, 1, (cuuint32_t)frames};
    CUtensorMap map;
    CTBB_TRY(tensor_map_f32(&map, p.raw, 4, dims, strides, box));
    CTBB_TRY(errors.ensure());
    int *err = errors.word;
    StagedRebin g;
    g.tiles = dt.tiles;
    g.n_tiles = (t.n_os + kRebinTile - 1) / kRebinTile;
    g.n_groups = (t.n_rows_raw + kRowsPerThread - 1) / kRowsPerThread;
    g.frames = frames;
    const int sides = (int)t.tiles.size() / g.n_tiles;
    const int chunks = (p.v_end - p.v_begin + kStagedViews - 1) / kStagedViews;
    const size_t smem = (size_t)(two ? 2 : 1) * frames * kRowsPerThread * channels * sizeof(float);
    const dim3 grid(g.n_tiles, g.n_groups * sides, chunks);
    auto launch = [&](auto kernel) -> int {
        CTBB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024));
        kernel<<<grid, 128, smem, stream>>>(p, g, map, err);
        count_launch();
        CTBB_CUDA_TRY(cudaGetLastError());
        return CTBB_OK;
    };
    if (channels == kNarrowBox)
        return two ? launch(rebin_staged_kernel<true, kNarrowBox>) : launch(rebin_staged_kernel<false, kNarrowBox>);
    return two ? launch(rebin_staged_kernel<true, kWideBox>) : launch(rebin_staged_kernel<false, kWideBox>);
}

int rebin_frames_needed(const RebinTables &t, int v)
{
    // view-axis coordinate of a focal spot's frame sequence: proj - t_alpha /
    // n_ffs - small focal terms, with |t_alpha| / n_ffs below the fan half
    // angle in views, which add_projections exceeds by 10; +1 for the upper
    // tap and one view of margin
    return t.n_ffs * (v + 2 * t.add_projections + 2);
}

int launch_rebin(const RebinTables &t, const DeviceRebinTables &dt, const float *d_raw,
                 float *d_out, CopyError &errors, cudaStream_t stream, int v_begin, int v_end)
{
    if (v_end < 0 || v_end > t.n_views) v_end = t.n_views;
    if (v_begin < 0) v_begin = 0;
    if (v_end <= v_begin) return CTBB_OK;
    RebinParams p;
    p.raw = d_raw;
    p.out = d_out;
    p.taps = dt.taps;
    p.focal = dt.focal;
    for (int i = 0; i < 4; ++i) p.focal_offset[i] = t.focal_offset[i];
    p.n_ffs = t.n_ffs;
    p.N = t.n_channels;
    p.Nos = t.n_os;
    p.R_raw = t.n_rows_raw;
    p.R = t.n_rows;
    p.n_proj = t.n_proj;
    p.add = t.add_projections;
    p.n_views = t.n_views;
    p.reverse_rows = t.reverse_rows;
    p.split_view_coord = t.split_view_coord;
    p.v_begin = v_begin;
    p.v_end = v_end;
    int chunks = (v_end - v_begin + kViewsPerThread - 1) / kViewsPerThread;
    int row_groups = (t.n_rows_raw + kRowsPerThread - 1) / kRowsPerThread;
    if (chunks > 65535 || row_groups > 65535) {
        set_error("rebin: %d views / %d rows exceed the launch grid", t.n_views, t.n_rows_raw);
        return CTBB_ERR_ARGUMENT;
    }
    const bool bilinear = t.mode == RebinMode::kNoFfs || t.mode == RebinMode::kZFfs;
    int channels = 0;
    if (const int frames = staged_frames(t, d_raw, bilinear ? 1 : 2, &channels))
        return launch_rebin_staged(t, dt, p, !bilinear, frames, channels, errors, stream);
    size_t n_raw = (size_t)t.n_ffs * t.n_proj * t.n_rows_raw * t.n_channels;
    size_t n_out = (size_t)t.n_views * t.n_rows * t.n_os;
    bool narrow = n_raw < ((size_t)1 << 31) && n_out < ((size_t)1 << 31);
    dim3 block(128);
    dim3 grid((t.n_os + 127) / 128, row_groups, chunks);
    if (bilinear && narrow) rebin_bilinear_kernel<int><<<grid, block, 0, stream>>>(p);
    else if (bilinear) rebin_bilinear_kernel<size_t><<<grid, block, 0, stream>>>(p);
    else if (narrow) rebin_two_stage_kernel<int><<<grid, block, 0, stream>>>(p);
    else rebin_two_stage_kernel<size_t><<<grid, block, 0, stream>>>(p);
    count_launch();
    CTBB_CUDA_TRY(cudaGetLastError());
    return CTBB_OK;
}

int upload_rebin_tables(const RebinTables &t, DeviceRebinTables *dt, cudaStream_t stream)
{
    size_t nt = t.out_taps.size() * sizeof(AxisTap);
    size_t nf = t.focal.size() * sizeof(FocalTerm), nb = t.tiles.size() * sizeof(RebinTile);
    if (dt->capacity < nt + nf + nb) {
        if (dt->base) cudaFree(dt->base);
        dt->base = nullptr;
        dt->capacity = 0;
        CTBB_CUDA_TRY(cudaMalloc(&dt->base, nt + nf + nb));
        dt->capacity = nt + nf + nb;
    }
    dt->taps = reinterpret_cast<AxisTap *>(dt->base);
    dt->focal = reinterpret_cast<FocalTerm *>(reinterpret_cast<char *>(dt->base) + nt);
    CTBB_CUDA_TRY(cudaMemcpyAsync(dt->taps, t.out_taps.data(), nt, cudaMemcpyHostToDevice, stream));
    dt->tiles = reinterpret_cast<RebinTile *>(reinterpret_cast<char *>(dt->base) + nt + nf);
    CTBB_CUDA_TRY(cudaMemcpyAsync(dt->focal, t.focal.data(), nf, cudaMemcpyHostToDevice, stream));
    CTBB_CUDA_TRY(cudaMemcpyAsync(dt->tiles, t.tiles.data(), nb, cudaMemcpyHostToDevice, stream));
    return CTBB_OK;
}

}  // namespace ctbb
