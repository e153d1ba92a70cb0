// backproject_staged.cu -- wFBP backprojection with the detector footprint of
// a CTA's voxel columns staged in shared memory.
//
// Same algorithm, arithmetic and border rules as the column form
// (backproject.cu); what differs is where the samples are read from and how
// the work is split.  A CTA owns 16 x 8 (or 8 x 8) voxel columns over the
// block's 32 slices; warp (cw, sg) owns the 8 x 4 columns cw and the 8 slices
// sg, whose image sums stay in registers.  A visit is a half-turn angle and a
// half turn whose rays reach the tile; the visits of a CTA are listed first,
// each with the box of detector rows and channels that the tile can touch and
// the class of every slice group, and packed into steps of at most four whose
// boxes fit half of a shared-memory buffer.  While a step is consumed from one
// half, the next step's boxes are copied into the other by TMA
// (cp.async.bulk.tensor, eight detector rows each, completion on an mbarrier),
// and slice group g computes the column geometry of its visit g.
//
// Why this split.  The column form is bound by the L1 data pipe (85 %: a 2x2
// footprint is four gathers whose lanes fall on two rows of the same banks)
// and close behind by issue (76 %).  Staged, the gathers take 1.2 wavefronts
// each (rows 24 banks apart), the image sums cost no shared memory, classes
// come from the visit list instead of votes, and the data pipe falls to 66 %;
// issue (77 %) and the wait for the slowest slice group of a step bound it.
// Measured on a 32-slice block against the column form (ms): 512^2, 1472 x 128
// rows, 3 half turns 12.10 -> 11.56; 512^2, 1472 x 64, 4 half turns 13.85 ->
// 12.69; 256^2, 1344 x 16, 6 half turns 3.98 -> 3.85; 333 x 259, 1344 x 64, 3
// half turns 3.26 -> 2.87.  A 48^2 block of 12 half turns, which the column
// form does not hold: 0.51 (slice-chunk form) -> 0.20.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <vector>

#include "backproject.h"
#include "backproject_box.cuh"
#include "backproject_device.cuh"
#include "ctbb_internal.h"
#include "cuda_util.cuh"
#include "tma.cuh"

namespace ctbb {

namespace {

constexpr int kRecords = 192;       // visits of one segment of angles
constexpr int kWideVisits = 608;    // staged_shape: most tiles x half turns of the 8 x 8 tile

// Shared memory of a CTA: the two halves of the box buffer, the column
// geometry of a step in each, the visits' records (four arrays), each step's
// plan words and first visit, the barriers and the record scan's warp counts.
struct StagedLayout {
    unsigned half_bytes, geo_w, geo_a, recs, plans, steps, bytes, bars, counts, total;
};

__host__ __device__ inline StagedLayout staged_layout(int cw, unsigned half_bytes)
{
    StagedLayout l;
    const unsigned cols = 32u * (unsigned)cw;
    l.half_bytes = half_bytes;
    l.geo_w = 2u * half_bytes;
    l.geo_a = l.geo_w + 2u * kGroups * cols * 16u;
    l.recs = l.geo_a + 2u * kGroups * cols * 4u;
    l.plans = l.recs + kRecords * 40u;
    l.steps = l.plans + kRecords * 16u;
    l.bytes = l.steps + (2u * kRecords + 4u) * 2u;
    l.bars = l.bytes + kRecords * 4u;
    l.counts = l.bars + 4u * 8u;
    l.total = l.counts + 32u * 4u;
    return l;
}

// kBoxRows rows of PITCH samples of the rows buffer seen as one matrix
__device__ __forceinline__ void tma_rows(uint32_t dst, const CUtensorMap *map, int x, int row, uint32_t bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(row), "r"(bar)
        : "memory");
}

// v of a warp whose lanes all hold the same value, in a form the compiler
// knows to be uniform (branches on it need no reconvergence)
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __reduce_or_sync(0xffffffffu, v); }

__device__ __forceinline__ bool elect_one()
{
    uint32_t yes;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(yes));
    return yes != 0;
}

template <int OFF>
__device__ __forceinline__ float lds_f32(uint32_t a)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFF));
    return v;
}

__device__ __forceinline__ float reciprocal_root(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float reciprocal(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

template <int CW, int PITCH, class Params>
__device__ __forceinline__ void backproject_staged_tile(const Params &p, int bx, int by, int ac, int n_ac,
                                                        int out_mode, const StagedLayout lay, const CUtensorMap *map, int *error)
{
    extern __shared__ __align__(128) char smem[];
    constexpr int COLS = 32 * CW, THREADS = COLS * kGroups, TX = tile_x(CW);
    constexpr unsigned ROW = (unsigned)PITCH * 4u;  // bytes of a box row
    constexpr unsigned BOX = ROW * kBoxRows;        // of a TMA copy
    const int tid = threadIdx.x, lane = tid & 31, warp = (int)uniform((uint32_t)tid >> 5);
    const int cw = warp % CW, sg = warp / CW, col = cw * 32 + lane;
    const int xi = bx * TX + (CW == 4 ? (cw & 1) * 8 : 0) + (lane & 7);
    const int yi = by * kTileY + (CW == 4 ? (cw >> 1) * 4 : cw * 4) + (lane >> 3);
    const bool inside = xi < p.nx && yi < p.ny;
    // voxel centres with the reference's float operations; a column outside
    // the image computes its edge column and writes nothing
    auto centre_x = [&](int i) { return __fadd_rn(__fmul_rn(p.pix_x, __fsub_rn((float)i, p.x_c)), p.x0); };
    auto centre_y = [&](int i) { return __fadd_rn(__fmul_rn(p.pix_y, __fsub_rn((float)i, p.y_c)), p.y0); };
    const float x = centre_x(min(xi, p.nx - 1)), y = centre_y(min(yi, p.ny - 1));
    const int nos = p.nos;
    const float zbase = __ldg(p.zpos);
    const float zc = (float)(sg * kSub);
    const float hr = p.half_rows;
    const float q_max_last = (float)(p.n_rows - 2);
    const uint32_t base = smem_address(smem);
    const uint32_t full = base + lay.bars;
    uint4 *recs = reinterpret_cast<uint4 *>(smem + lay.recs);  // {row index, channels, rows, box offset}
    float4 *rec_t = reinterpret_cast<float4 *>(recs + kRecords);  // sin, cos, ray term; sin of the angle's k = 0 view
    float *rec_c0 = reinterpret_cast<float *>(rec_t + kRecords);  // cos of the angle's k = 0 view
    // classes of the slice groups | angle of the segment << 16 | last of its angle << 31
    uint32_t *rec_cls = reinterpret_cast<uint32_t *>(rec_c0 + kRecords);
    unsigned short *steps = reinterpret_cast<unsigned short *>(smem + lay.steps), *next = steps + kRecords + 2;
    // step n's plan for slice group g, plans[4 n + g]: 4 bits per visit (class,
    // 8 at the end of its angle), visits << 16, first visit << 24
    uint32_t *plans = reinterpret_cast<uint32_t *>(smem + lay.plans);
    uint32_t *step_bytes = reinterpret_cast<uint32_t *>(smem + lay.bytes);
    const uint32_t geo_w = base + lay.geo_w + (uint32_t)col * 16u, geo_a = base + lay.geo_a + (uint32_t)col * 4u;
    int *counts = reinterpret_cast<int *>(smem + lay.counts);
    if (tid == 0) {
        barrier_init(full, 1);
        barrier_init(full + 8u, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }

    // This warp's share of a step (its plan), the g-th of the CTA, into half
    // g & 1: its columns' geometry of the step's visit sg and every CW-th copy
    // of that visit's box.  Entry of a column: {q0, dq, (1 - wp) c, wp c}, c =
    // [p on the detector], and the shared-memory address of (ip, row 0)
    // moved back as in row_floor.
    auto produce = [&](uint32_t plan, uint32_t bytes, uint32_t g) {
        const uint32_t half = g & 1u;
        if ((uint32_t)sg < (plan >> 16 & 7u)) {
            const int u = (int)(plan >> 24) + sg;
            const uint4 r = recs[u];
            const int ch0 = (int)r.y, row0 = (int)(r.z & 0xffffu);
            const uint32_t box = base + half * lay.half_bytes + r.w;
            // copy j of the box by column warp j % CW
            const uint32_t n_copies = uniform(r.z >> 16), dst = uniform(box);
            const int cx = (int)uniform((uint32_t)ch0);
            const int cy = (int)uniform(r.x * (unsigned)p.n_rows + (unsigned)row0);
            for (uint32_t j = (uint32_t)cw; j < n_copies; j += CW)
                if (elect_one()) tma_rows(dst + j * BOX, map, cx, cy + (int)j * kBoxRows, full + 8u * half);
            const float4 t = rec_t[u];
            const float t0_cos = rec_c0[u];
            // the angle's asin and root, carried to this half turn to first
            // order (see backproject_tile)
            const float phat0 = __fsub_rn(__fmul_rn(x, t.w), __fmul_rn(y, t0_cos));
            const float a_abs = fabsf(asin_fast(phat0 * p.inv_rf));
            const float l2 = fmaf(-phat0, phat0, p.rf2);
            const float inv_root = reciprocal_root(l2), root = l2 * inv_root, p0_abs = fabsf(phat0);
            const float slope = p0_abs * inv_root;
            const float a_off = fmaf(-p0_abs, inv_root, a_abs), root_off = fmaf(slope, p0_abs, root);
            const float phat = __fsub_rn(__fmul_rn(x, t.x), __fmul_rn(y, t.y));
            const float a_k = fmaf(fabsf(phat), inv_root, a_off);
            const float root_k = fmaf(-slope, fabsf(phat), root_off);
            const float zb_ray = fmaf(copysignf(a_k, phat), p.zrot_over_2pi, zbase - t.z);
            const float lhat = root_k - x * t.y - y * t.x;
            const float inv_den = reciprocal(lhat * p.tan_cone);
            const float p_max = (float)(nos - 2), p_mid = 0.5f * p_max;
            float p_idx = fmaf(phat, p.inv_ds_half, p.two_cc);
            if (fabsf(p_idx - p_mid) > p_mid - kBorderBand) p_idx = p_index_exact(p, phat);
            const bool p_ok = (p_idx >= 0.0f) && (p_idx <= p_max);
            const int ip = p_ok ? (int)p_idx : (p_idx < 0.0f ? 0 : nos - 2);
            const float wp = p_idx - (float)ip;
            const float c = p_ok ? 1.0f : 0.0f;
            const uint32_t e = half * kGroups + (uint32_t)sg;
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(geo_w + e * (COLS * 16u)),
                         "f"(zb_ray * inv_den), "f"(p.coll * inv_den), "f"((1.0f - wp) * c), "f"(wp * c)
                         : "memory");
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(geo_a + e * (COLS * 4u)),
                         "r"(box + (uint32_t)(ip - ch0) * 4u - ((uint32_t)row0 + kFloorMagicBits) * ROW)
                         : "memory");
        }
        if (warp == 0 && elect_one()) barrier_arrive_expect(full + 8u * half, bytes);
    };

    float2 img[kSub / 2], s2[kSub / 2], h2[kSub / 2];
#pragma unroll
    for (int m = 0; m < kSub / 2; ++m) img[m] = s2[m] = h2[m] = make_float2(0.0f, 0.0f);
    const int i_begin = (int)(((long long)ac * p.n_half) / n_ac);
    const int i_end = (int)(((long long)(ac + 1) * p.n_half) / n_ac);
    const int seg = kRecords / p.nht;
    uint32_t use = 0;  // steps consumed, over all segments
    bool alive = true;
    for (int ia = i_begin; ia < i_end; ia += seg) {
        // the segment's visits, in order
        __syncthreads();
        const int n_slots = min(seg, i_end - ia) * p.nht;
        uint32_t chan = 0, rows = 0, cls = 0;
        float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        bool need = false;
        const int vi = ia + tid / p.nht, vk = tid % p.nht;
        if (tid < n_slots) {
            const float xa = centre_x(bx * TX), xb = centre_x(min(bx * TX + TX - 1, p.nx - 1));
            const float ya = centre_y(by * kTileY), yb = centre_y(min(by * kTileY + kTileY - 1, p.ny - 1));
            t = __ldg(p.views + (size_t)vi * p.nht + vk);
            need = visit_box(p, t, vk == p.nht - 1, zbase, 0.5f * (xa + xb), 0.5f * fabsf(xb - xa) + 1e-3f,
                             0.5f * (ya + yb), 0.5f * fabsf(yb - ya) + 1e-3f, &chan, &rows, &cls);
        }
        const unsigned ballot = __ballot_sync(0xffffffffu, need);
        if (lane == 0) counts[warp] = __popc(ballot);
        __syncthreads();
        int at = __popc(ballot & ((1u << lane) - 1u)), n_visits = 0;
        for (int w = 0; w < THREADS / 32; ++w) {
            if (w < warp) at += counts[w];
            n_visits += counts[w];
        }
        if (need) {
            const float4 t0 = __ldg(p.views + (size_t)vi * p.nht);
            recs[at] = make_uint4(__float_as_uint(t.x), chan, rows, 0u);
            rec_t[at] = make_float4(t.y, t.z, t.w, t0.y);
            rec_c0[at] = t0.z;
            rec_cls[at] = cls | (uint32_t)(vi - ia) << 16;
        }
        __syncthreads();
        // Steps: consecutive visits whose boxes fit a half, at most four.
        // Every visit finds the end of a step beginning at it, one thread
        // follows the ends, and each step then places its boxes.
        bool ends = false;
        if (tid < n_visits) {
            uint32_t used = recs[tid].z >> 16;
            int end = tid + 1;
            while (end < n_visits && end < tid + kGroups && (used + (recs[end].z >> 16)) * BOX <= lay.half_bytes)
                used += recs[end++].z >> 16;
            next[tid] = (unsigned short)end;
            ends = tid + 1 == n_visits || rec_cls[tid] >> 16 != rec_cls[tid + 1] >> 16;
        }
        __syncthreads();
        if (ends) rec_cls[tid] |= 0x80000000u;
        if (tid == 0) {
            int n = 0;
            for (int v = 0; v < n_visits; v = next[v]) steps[n++] = (unsigned short)v;
            steps[n] = (unsigned short)n_visits;
            counts[31] = n;
        }
        __syncthreads();
        const int n_steps = (int)uniform((uint32_t)counts[31]);
        if (tid < n_steps) {
            const int first = steps[tid], end = steps[tid + 1];
            uint32_t used = 0, words[kGroups] = {};
            for (int v = first; v < end; ++v) {
                recs[v].w = used;
                used += (recs[v].z >> 16) * BOX;
                const uint32_t c = rec_cls[v];
                for (int g = 0; g < kGroups; ++g) words[g] |= ((c >> (3 * g) & 7u) | (c >> 31 << 3)) << (4 * (v - first));
            }
            step_bytes[tid] = used;
            for (int g = 0; g < kGroups; ++g)
                plans[tid * kGroups + g] = words[g] | (uint32_t)(end - first) << 16 | (uint32_t)first << 24;
        }
        __syncthreads();

        float n_flat = 1e-30f;
        // two steps ahead of their consumption
        uint32_t plan = 0, plan_next = 0;
        if (n_steps > 0) {
            plan = uniform(plans[sg]);
            produce(plan, step_bytes[0], use);
        }
        if (n_steps > 1) {
            plan_next = uniform(plans[kGroups + sg]);
            produce(plan_next, step_bytes[1], use + 1u);
        }
        __syncthreads();
        for (int n = 0; n < n_steps; ++n, ++use) {
            const uint32_t half = use & 1u;
            const uint32_t ahead = n + 2 < n_steps ? uniform(plans[(n + 2) * kGroups + sg]) : 0u;
            alive = barrier_wait(full + 8u * half, use >> 1 & 1u);
            const int v0 = (int)(plan >> 24), n_visits_step = (int)(plan >> 16 & 7u);
            uint32_t gw = geo_w + half * (kGroups * COLS * 16u), ga = geo_a + half * (kGroups * COLS * 4u);
            for (int j = 0; j < n_visits_step; ++j, plan >>= 4, gw += COLS * 16u, ga += COLS * 4u) {
                const uint32_t kind = plan & 7u;
                if (kind != kSkip) {
                    float4 g;
                    uint32_t addr;
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                 : "=f"(g.x), "=f"(g.y), "=f"(g.z), "=f"(g.w)
                                 : "r"(gw));
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(addr) : "r"(ga));
                    const float2 wp2 = make_float2(g.w, g.w), omwp2 = make_float2(g.z, g.z);
                    const float2 dq2 = make_float2(g.y, g.y), q02 = make_float2(g.x, g.x), hr2 = make_float2(hr, hr);
                    // cos^2 taper weight of a pair: W = 1 below Q (cos(0) = 1), then
                    // cos^2(pi/2 (|q| - Q) / (1 - Q))
                    auto pair_weight = [&](float2 q) -> float2 {
                        const float2 a = fma2(make_float2(fmaxf(fabsf(q.x), kQ), fmaxf(fabsf(q.y), kQ)),
                                              make_float2(p.taper_scale, p.taper_scale),
                                              make_float2(-kQ * p.taper_scale, -kQ * p.taper_scale));
                        const float2 cc = make_float2(__cosf(a.x), __cosf(a.y));
                        return mul2(cc, cc);
                    };
                    auto slice_pair = [&](int m) { return make_float2(zc + (float)(2 * m), zc + (float)(2 * m + 1)); };
                    auto fetch = [&](float tr, float &v00, float &v01, float &v10, float &v11) {
                        const uint32_t o = addr + __float_as_uint(tr) * ROW;
                        v00 = lds_f32<0>(o), v01 = lds_f32<4>(o);
                        v10 = lds_f32<(int)ROW>(o), v11 = lds_f32<(int)ROW + 4>(o);
                    };
                    // bilinear value of a pair of row coordinates ql, tr their floors
                    auto pair_value = [&](float2 ql, float2 tr) -> float2 {
                        const float2 wq = sub2(ql, sub2(tr, make_float2(kFloorMagic, kFloorMagic)));
                        float a00, a01, a10, a11, b00, b01, b10, b11;
                        fetch(tr.x, a00, a01, a10, a11);
                        fetch(tr.y, b00, b01, b10, b11);
                        const float2 c0 = fma2(wp2, make_float2(a01, b01), mul2(omwp2, make_float2(a00, b00)));
                        const float2 c1 = fma2(wp2, make_float2(a11, b11), mul2(omwp2, make_float2(a10, b10)));
                        return fma2(wq, sub2(c1, c0), c0);
                    };
                    if (kind == kFlat) {
                        const float ql0 = fmaf(g.x, hr, hr), dql = g.y * hr;
                        const float2 ql02 = make_float2(ql0, ql0), dql2 = make_float2(dql, dql);
#pragma unroll
                        for (int m = 0; m < kSub / 2; ++m) {
                            const float2 ql = fma2(slice_pair(m), dql2, ql02);
                            s2[m] = add2(s2[m], pair_value(ql, row_floor(ql)));
                        }
                        n_flat += 1.0f;
                    } else if (kind == kInner) {
#pragma unroll
                        for (int m = 0; m < kSub / 2; ++m) {
                            const float2 q = fma2(slice_pair(m), dq2, q02);
                            const float2 ql = fma2(q, hr2, hr2);
                            const float2 w = pair_weight(q);
                            h2[m] = add2(h2[m], w);
                            s2[m] = fma2(w, pair_value(ql, row_floor(ql)), s2[m]);
                        }
                    } else if (kind == kOther) {
                        const float t_max = kFloorMagic + (float)(p.n_rows - 2);  // row R-2
#pragma unroll
                        for (int m = 0; m < kSub / 2; ++m) {
                            const float2 q = fma2(slice_pair(m), dq2, q02);
                            const bool in_x = fabsf(q.x) < 1.0f, in_y = fabsf(q.y) < 1.0f;
                            if (!__any_sync(0xffffffffu, in_x || in_y)) continue;
                            float2 w = pair_weight(q);
                            w = make_float2(in_x ? w.x : 0.0f, in_y ? w.y : 0.0f);
                            h2[m] = add2(h2[m], w);
                            const float2 ql = fma2(q, hr2, hr2);
                            float2 tr = row_floor(ql);
                            tr = make_float2(fminf(fmaxf(tr.x, kFloorMagic), t_max),
                                             fminf(fmaxf(tr.y, kFloorMagic), t_max));
                            s2[m] = fma2(w, pair_value(ql, tr), s2[m]);
                        }
                    } else if (kind == kOff) {
#pragma unroll
                        for (int m = 0; m < kSub / 2; ++m) {
                            const float2 q = fma2(slice_pair(m), dq2, q02);
                            const float2 w = pair_weight(q);
                            h2[m] = add2(h2[m], make_float2(fabsf(q.x) < 1.0f ? w.x : 0.0f,
                                                            fabsf(q.y) < 1.0f ? w.y : 0.0f));
                        }
                    } else {
                        // rare: rows near the last half turn's border, decided by
                        // the reference's own q_idx
                        const float t_max = kFloorMagic + (float)(p.n_rows - 2);
                        const size_t view = (size_t)(ia + (int)(rec_cls[v0 + j] >> 16 & 0x7fffu)) * p.nht + (p.nht - 1);
                        const float4 tv = __ldg(p.views + view);
                        const float theta = __ldg(p.theta + view);
                        const float phat = __fsub_rn(__fmul_rn(x, tv.y), __fmul_rn(y, tv.z));
                        const bool p_ok = (g.z != 0.0f) || (g.w != 0.0f);
#pragma unroll 1
                        for (int m = 0; m < kSub; ++m) {
                            const float q = fmaf(zc + (float)m, g.y, g.x);
                            const bool in = fabsf(q) < 1.0f;
                            const float w = in ? pair_weight(make_float2(q, q)).x : 0.0f;
                            const float ql = fmaf(q, hr, hr);
                            const float tr = fminf(fmaxf(__fadd_rd(ql, kFloorMagic), kFloorMagic), t_max);
                            const float val = pair_value(make_float2(ql, ql), make_float2(tr, tr)).x;
                            const float d = ql - q_max_last;
                            bool kept = in && p_ok && !(d > kBorderBand);
                            if (kept && d > -kBorderBand)
                                kept = last_turn_sample_valid(p, x, y, theta, tv.y, tv.z, phat,
                                                              __ldg(p.zpos + min(sg * kSub + m, p.n_slices - 1)),
                                                              p.nht - 1);
                            const float wv = kept ? w : 0.0f;
#pragma unroll
                            for (int j = 0; j < kSub / 2; ++j) {
                                if (m == 2 * j) {
                                    h2[j].x += w;
                                    s2[j].x = fmaf(wv, val, s2[j].x);
                                } else if (m == 2 * j + 1) {
                                    h2[j].y += w;
                                    s2[j].y = fmaf(wv, val, s2[j].y);
                                }
                            }
                        }
                    }
                }
                if (plan & 8u) {
                    // the angle's last visit: image += s / h.  s is 0 wherever h
                    // is; n_flat starts at 1e-30, far below the smallest nonzero
                    // weight, so that such a quotient is 0
#pragma unroll
                    for (int m = 0; m < kSub / 2; ++m) {
                        const float2 hz = add2(h2[m], make_float2(n_flat, n_flat));
                        img[m] = fma2(s2[m], make_float2(reciprocal(hz.x), reciprocal(hz.y)), img[m]);
                        s2[m] = h2[m] = make_float2(0.0f, 0.0f);
                    }
                    n_flat = 1e-30f;
                }
            }
            // every warp is done with this half (and has read its waits'
            // outcome: one that ran out ends the CTA)
            if (__syncthreads_or(!alive)) {
                alive = false;
                break;
            }
            if (n + 2 < n_steps) produce(ahead, step_bytes[n + 2], use + 2u);
            plan = plan_next;
            plan_next = ahead;
        }
        if (!alive) break;
    }
    if (!alive) {
        // a wait ran out: report it, and no image in place of a part of one
        *reinterpret_cast<volatile int *>(error) = 1;
        wait_for_stray_copies();
#pragma unroll
        for (int m = 0; m < kSub / 2; ++m)
            img[m] = make_float2(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
    }
    if (!inside) return;
    const size_t plane = (size_t)p.nx * p.ny;
    float *dst = out_mode == kOutPartial ? p.partial + (size_t)ac * p.n_slices * plane : p.out;
    dst += (size_t)yi * p.nx + xi;
#pragma unroll
    for (int m = 0; m < kSub; ++m) {
        const int z = sg * kSub + m;
        if (z >= p.n_slices) break;
        const float v = (m & 1) ? img[m / 2].y : img[m / 2].x;
        float *o = dst + (size_t)z * plane;
        switch (out_mode) {
        case kOutScaled: *o = v * p.out_scale; break;
        case kOutMiddle: *o = *o + v; break;
        case kOutLast: *o = (*o + v) * p.out_scale; break;
        default: *o = v;  // kOutPartial, kOutFirst
        }
    }
}

// 64 registers: 1024 threads per SM.
template <int CW, int PITCH>
__global__ void __launch_bounds__(128 * CW, 8 / CW) backproject_staged_kernel(BpParams p, StagedLayout lay, const __grid_constant__ CUtensorMap map, int *error)
{
    backproject_staged_tile<CW, PITCH>(p, blockIdx.x, blockIdx.y, blockIdx.z, p.n_achunks,
                                             p.partial ? kOutPartial : kOutScaled, lay, &map, error);
}

// The blocks of a batch in one launch per angle chunk (see
// backproject_column_batch_kernel), or, ac < 0, with grid y over the chunks,
// which write partial sums.
template <int CW, int PITCH>
__global__ void __launch_bounds__(128 * CW, 8 / CW)
    backproject_staged_batch_kernel(const BpParams *__restrict__ params, const unsigned *__restrict__ tile_start,
                                    const CUtensorMap *__restrict__ maps, int n_blocks, int ac, int n_ac,
                                    StagedLayout lay, int *error)
{
    __shared__ BpParams sp;
    __shared__ int s_block;
    const unsigned tile = blockIdx.x;
    if (threadIdx.x == 0) {
        int lo = 0, hi = n_blocks - 1;  // the last b with tile_start[b] <= tile
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(tile_start + mid) <= tile) lo = mid;
            else hi = mid - 1;
        }
        s_block = lo;
    }
    __syncthreads();
    const int b = s_block;
    const uint32_t *src = reinterpret_cast<const uint32_t *>(params + b);
    uint32_t *dst = reinterpret_cast<uint32_t *>(&sp);
    for (int w = threadIdx.x; w < (int)(sizeof(BpParams) / 4); w += 128 * CW) dst[w] = __ldg(src + w);
    __syncthreads();
    // the map was written by a copy before this launch
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(reinterpret_cast<uint64_t>(maps + b))
                 : "memory");
    const unsigned local = tile - __ldg(tile_start + b);
    const unsigned gx = (unsigned)((sp.nx + tile_x(CW) - 1) / tile_x(CW));
    const int mode = ac < 0      ? kOutPartial
                     : n_ac == 1 ? kOutScaled
                     : ac == 0   ? kOutFirst
                                 : (ac == n_ac - 1 ? kOutLast : kOutMiddle);
    backproject_staged_tile<CW, PITCH>(sp, (int)(local % gx), (int)(local / gx), ac < 0 ? (int)blockIdx.y : ac, n_ac,
                                             mode, lay, maps + b, error);
}

// Calls f(CW, PITCH) with a shape's compile-time instance.
template <class F>
int with_staged(const StagedShape &s, F &&f)
{
    using std::integral_constant;
    if (s.cw == 4 && s.pitch == 56) return f(integral_constant<int, 4>(), integral_constant<int, 56>());
    if (s.cw == 4 && s.pitch == 88) return f(integral_constant<int, 4>(), integral_constant<int, 88>());
    if (s.cw == 2 && s.pitch == 88) return f(integral_constant<int, 2>(), integral_constant<int, 88>());
    set_error("backproject: no staged kernel for %d column warps, rows of %d", s.cw, s.pitch);
    return CTBB_ERR_ARGUMENT;
}

// The rows buffer of a block as a matrix of view rows, box kBoxRows x pitch
// samples; samples past its edges read as zeros.
int rows_map(const BpParams &p, int pitch, CUtensorMap *map)
{
    const cuuint64_t dims[2] = {(cuuint64_t)p.nos, (cuuint64_t)p.n_views * (cuuint64_t)p.n_rows};
    const cuuint64_t strides[1] = {dims[0] * 4};
    const cuuint32_t box[2] = {(cuuint32_t)pitch, (cuuint32_t)kBoxRows};
    return tensor_map_f32(map, p.rebin, 2, dims, strides, box);
}

int raise_smem_limit(const void *kernel)
{
    CTBB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024));
    return CTBB_OK;
}

}  // namespace

bool staged_shape(const BpParams &p, StagedShape *out)
{
    // FP32 rows (FP16 footprint words: 8 bytes a sample, twice the copies, took
    // 2.9 -> 3.9 ms per block); TMA copies start on 16-byte boundaries
    if (p.vscale || p.nos % 4 != 0 || ((uintptr_t)p.rebin & 15) != 0) return false;
    if (p.n_slices > kGroups * kSub || p.nht > kRecords || p.n_half > 65535 || p.nos > 65535 || p.n_rows > 4096)
        return false;
    if (!(p.coll > 0.0f)) return false;
    if ((double)p.n_views * (double)p.n_rows >= 2147483648.0) return false;
    // every voxel well inside the source's circle
    const float rx = std::fabs(p.x0) + 0.5f * std::fabs(p.pix_x) * (float)p.nx;
    const float ry = std::fabs(p.y0) + 0.5f * std::fabs(p.pix_y) * (float)p.ny;
    if (!(std::sqrt(rx * rx + ry * ry) < 0.9f * p.rf)) return false;
    // Beyond the column form's windows the alternative is the slice-chunk form.
    // A visit is staged for whole groups of 8 slices; where the detector spans
    // fewer, most of that is idle, which small images repay (the slice-chunk
    // form has too few CTAs for them) and large ones do not.  ms against the
    // slice-chunk form, by the slices between the detector's edges at the
    // isocentre and tiles of 16 x 8: 1 slice, 50 tiles 0.55 / 0.89, 120 1.11 /
    // 1.00, 512 4.26 / 2.68; 3 slices, 50 0.40 / 0.81, 120 0.81 / 0.90, 190
    // 1.21 / 1.03, 512 3.09 / 2.48; 7 slices, 325 2.08 / 2.29, 512 3.11 / 3.10,
    // 1152 6.81 / 6.23; 15 slices, 1152 5.24 / 6.05.
    if (p.nht > kColumnMaxHalfTurns) {
        const float seen = 2.0f * p.rf * p.tan_cone / p.coll;
        const long long tiles = (long long)((p.nx + 15) / 16) * ((p.ny + kTileY - 1) / kTileY);
        if (!(seen >= 12.0f) && tiles > (seen >= 6.0f ? 448 : 96)) return false;
    }
    struct Candidate {
        int cw, pitch;
    };
    for (const Candidate c : {Candidate{4, 56}, Candidate{4, 88}, Candidate{2, 88}}) {
        const float wx = (float)(tile_x(c.cw) - 1) * std::fabs(p.pix_x), wy = (float)(kTileY - 1) * std::fabs(p.pix_y);
        const float span = (std::sqrt(wx * wx + wy * wy) + 4e-3f) * std::fabs(p.inv_ds_half) + 2.0f * kBoxMargin + 0.01f;
        if (!(span < 1000.0f)) continue;
        // visit_box bounds p and the ray position of a tile separately: the
        // rectangle they span around the tile has to lie inside the source's
        // circle too, or its distances to the source turn negative
        // (tiles of tens of centimetres, on detectors of few channels)
        const float hx = 0.5f * (float)(std::min(tile_x(c.cw), p.nx) - 1) * std::fabs(p.pix_x);
        const float hy = 0.5f * (float)(std::min(kTileY, p.ny) - 1) * std::fabs(p.pix_y);
        const float tx = rx - hx, ty = ry - hy;  // the outermost tile's centre
        if (!(std::sqrt(tx * tx + ty * ty) + hx + hy < 0.95f * p.rf)) continue;
        // Coarse pixels (8 x 8 tiles, wide boxes) copy more per voxel than the
        // column form gathers; their four warps per 32 columns pay where the
        // column form has too few CTAs, or does not hold the window.  ms
        // against the column form, by tiles x half turns: 93^2, 576: 0.47 /
        // 0.78; 109^2, 588: 0.53 / 0.69; 133 x 99, 884: 0.35 / 0.30; 118^2,
        // 1125: 0.83 / 0.80; 171^2, 2420: 1.89 / 1.66; 231 x 207, 3016: 3.63 /
        // 3.29.
        if (c.cw == 2 && p.nht <= kColumnMaxHalfTurns &&
            ((p.nx + 7) / 8) * ((p.ny + kTileY - 1) / kTileY) * p.nht > kWideVisits)
            continue;
        // channels from the first, moved down to a multiple of 4, to the one past the last
        if ((int)std::floor(span) + 3 + 3 > c.pitch) continue;
        // the whole of a view's rows fits a half, and at most four of them are
        // of use; shared memory for 1024 threads per SM, else for 512
        const unsigned box = (unsigned)((p.n_rows + kBoxRows - 1) / kBoxRows * kBoxRows * c.pitch) * 4u;
        const unsigned rest = staged_layout(c.cw, 0).total;
        for (unsigned ctas : {8u / (unsigned)c.cw, 4u / (unsigned)c.cw}) {
            const unsigned limit = (227u * 1024u) / ctas - 1024u - 512u;
            if (limit < rest) continue;
            const unsigned half = std::min((limit - rest) / 2u & ~127u, kGroups * box);
            if (half < box) continue;
            out->cw = c.cw;
            out->pitch = c.pitch;
            out->half_bytes = half;
            return true;
        }
    }
    return false;
}

int launch_backproject_staged(const BpParams &p, const StagedShape &s, CopyError &errors, cudaStream_t stream)
{
    CTBB_TRY(errors.ensure());
    int *err = errors.word;
    const dim3 grid((p.nx + tile_x(s.cw) - 1) / tile_x(s.cw), (p.ny + kTileY - 1) / kTileY, std::max(p.n_achunks, 1));
    return with_staged(s, [&](auto cw, auto pitch) -> int {
        constexpr int CW = decltype(cw)::value, PITCH = decltype(pitch)::value;
        const StagedLayout lay = staged_layout(CW, s.half_bytes);
        CUtensorMap map;
        CTBB_TRY(rows_map(p, PITCH, &map));
        CTBB_TRY(raise_smem_limit(reinterpret_cast<const void *>(backproject_staged_kernel<CW, PITCH>)));
        backproject_staged_kernel<CW, PITCH><<<grid, 128 * CW, lay.total, stream>>>(p, lay, map, err);
        count_launch();
        CTBB_CUDA_TRY(cudaGetLastError());
        return CTBB_OK;
    });
}

int staged_chunks(const BpParams &p, const StagedShape &s, int limit)
{
    return staged_tiles(p, s) >= 304u ? std::max(1, limit / 2) : limit;
}

unsigned staged_tiles(const BpParams &p, const StagedShape &s)
{
    return (unsigned)((p.nx + tile_x(s.cw) - 1) / tile_x(s.cw)) * (unsigned)((p.ny + kTileY - 1) / kTileY);
}

size_t staged_map_bytes() { return sizeof(CUtensorMap); }

int staged_map(const BpParams &p, const StagedShape &s, void *out)
{
    return rows_map(p, s.pitch, static_cast<CUtensorMap *>(out));
}

int launch_backproject_staged_batch(const BpParams *d_params, const unsigned *d_start, const void *d_maps,
                                    unsigned total, int n, int ac, int n_ac, const StagedShape &s,
                                    CopyError &errors, cudaStream_t stream)
{
    CTBB_TRY(errors.ensure());
    int *err = errors.word;
    return with_staged(s, [&](auto cw, auto pitch) -> int {
        constexpr int CW = decltype(cw)::value, PITCH = decltype(pitch)::value;
        const StagedLayout lay = staged_layout(CW, s.half_bytes);
        CTBB_TRY(raise_smem_limit(reinterpret_cast<const void *>(backproject_staged_batch_kernel<CW, PITCH>)));
        backproject_staged_batch_kernel<CW, PITCH>
            <<<dim3(total, ac < 0 ? n_ac : 1), 128 * CW, lay.total, stream>>>(
                d_params, d_start, static_cast<const CUtensorMap *>(d_maps), n, ac, n_ac, lay, err);
        count_launch();
        CTBB_CUDA_TRY(cudaGetLastError());
        return CTBB_OK;
    });
}

}  // namespace ctbb
