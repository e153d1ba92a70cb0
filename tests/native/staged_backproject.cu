// Host check of the staged backprojector's boxes: for the tiles, angles and
// half turns of a planned block, every detector sample that the kernel
// addresses for a column of the tile against the box it would copy, and every
// slice against the class its group was given.  The columns' geometry is the
// kernel's (asin and root carried from the angle's first half turn to first
// order), with the host's functions.
#include <cmath>
#include <cstdint>
#include <vector>

#include "backproject.h"
#include "backproject_box.cuh"

using namespace ctbb;

namespace {

int block_params(const struct recon_metadata *mr, BackprojectTables *t, BpParams *p)
{
    const int st = build_backproject_tables(*mr, t);
    if (st) return st;
    alignas(16) static const float rows[4] = {};
    return make_backproject_params(*mr, *t, reinterpret_cast<const float4 *>(t->views.data()), t->theta.data(),
                                   t->zpos.data(), rows, nullptr, nullptr, BpShape{}, p);
}

}  // namespace

// The staged form's tile of a block: column warps and box pitch (0, 0 where
// another form runs).
extern "C" int check_staged_shape(const struct recon_metadata *mr, int *cw, int *pitch)
{
    BackprojectTables t;
    BpParams p;
    const int st = block_params(mr, &t, &p);
    if (st) return st;
    StagedShape s;
    *cw = *pitch = 0;
    if (staged_shape(p, &s)) *cw = s.cw, *pitch = s.pitch;
    return CTBB_OK;
}

// Visits looked at in *visits (0: not staged), samples addressed outside their
// box in *outside, slices that their group's class does not hold for in
// *misread.  Every angle_step-th angle.
extern "C" int check_staged_boxes(const struct recon_metadata *mr, int angle_step, long long *visits,
                                  long long *outside, long long *misread)
{
    BackprojectTables t;
    BpParams p;
    const int st = block_params(mr, &t, &p);
    if (st) return st;
    *visits = *outside = *misread = 0;
    StagedShape s;
    if (!staged_shape(p, &s)) return CTBB_OK;
    const int TX = tile_x(s.cw);
    auto centre_x = [&](int i) { return p.pix_x * ((float)i - p.x_c) + p.x0; };
    auto centre_y = [&](int i) { return p.pix_y * ((float)i - p.y_c) + p.y0; };
    const float zbase = p.zpos[0];
    for (int by = 0; by * kTileY < p.ny; ++by)
        for (int bx = 0; bx * TX < p.nx; ++bx) {
            const int x1 = std::min(bx * TX + TX - 1, p.nx - 1), y1 = std::min(by * kTileY + kTileY - 1, p.ny - 1);
            const float xa = centre_x(bx * TX), xb = centre_x(x1), ya = centre_y(by * kTileY), yb = centre_y(y1);
            for (int i = 0; i < p.n_half; i += angle_step)
                for (int k = 0; k < p.nht; ++k) {
                    const float4 t0 = p.views[(size_t)i * p.nht], v = p.views[(size_t)i * p.nht + k];
                    uint32_t chan = 0, rows = 0, cls = 0;
                    const bool last = k == p.nht - 1;
                    const bool need = visit_box(p, v, last, zbase, 0.5f * (xa + xb), 0.5f * std::fabs(xb - xa) + 1e-3f,
                                                0.5f * (ya + yb), 0.5f * std::fabs(yb - ya) + 1e-3f, &chan, &rows,
                                                &cls);
                    ++*visits;
                    const int row0 = (int)(rows & 0xffffu), n_rows = (int)(rows >> 16) * kBoxRows;
                    for (int yi = by * kTileY; yi <= y1; ++yi)
                        for (int xi = bx * TX; xi <= x1; ++xi) {
                            const float x = centre_x(xi), y = centre_y(yi);
                            const float phat0 = x * t0.y - y * t0.z, a_abs = std::fabs(std::asin(phat0 * p.inv_rf));
                            const float l2 = p.rf2 - phat0 * phat0, root = std::sqrt(l2), inv_root = 1.0f / root;
                            const float p0_abs = std::fabs(phat0), slope = p0_abs * inv_root;
                            const float phat = x * v.y - y * v.z;
                            const float a_k = a_abs + (std::fabs(phat) - p0_abs) * inv_root;
                            const float root_k = root - slope * (std::fabs(phat) - p0_abs);
                            const float zb = std::copysign(a_k, phat) * p.zrot_over_2pi + (zbase - v.w);
                            const float inv_den = 1.0f / ((root_k - x * v.z - y * v.y) * p.tan_cone);
                            const float q0 = zb * inv_den, dq = p.coll * inv_den;
                            const float p_idx = phat * p.inv_ds_half + p.two_cc;
                            const bool p_ok = p_idx >= 0.0f && p_idx <= (float)(p.nos - 2);
                            const int ip = p_ok ? (int)p_idx : (p_idx < 0.0f ? 0 : p.nos - 2);
                            for (int z = 0; z < kGroups * kSub; ++z) {
                                const float q = q0 + (float)z * dq, ql = q * p.half_rows + p.half_rows;
                                const bool in = std::fabs(q) < 1.0f && z < p.n_slices;
                                const uint32_t kind = need ? cls >> (3 * (z / kSub)) & 7u : (uint32_t)kSkip;
                                if (kind == kSkip) {
                                    if (in) ++*misread;
                                    continue;
                                }
                                if (kind == kOff) {
                                    if (p_ok) ++*misread;
                                    continue;
                                }
                                // a class holds for the group's 8 slices, also past the block's end
                                if (kind == kFlat && std::fabs(q) > kQ) ++*misread;
                                if (kind == kInner && (std::fabs(q) >= 1.0f || (last && ql > (float)(p.n_rows - 2))))
                                    ++*misread;
                                if (kind == kOther && last && in && ql > (float)(p.n_rows - 2)) ++*misread;
                                float tr = std::floor(ql);
                                if (kind == kOther || kind == kBorder)
                                    tr = std::fmin(std::fmax(tr, 0.0f), (float)(p.n_rows - 2));
                                if (!(tr >= (float)row0 && tr + 1.0f < (float)(row0 + n_rows))) ++*outside;
                                if (ip < (int)chan || ip + 1 >= (int)chan + s.pitch) ++*outside;
                            }
                        }
                }
        }
    return CTBB_OK;
}
