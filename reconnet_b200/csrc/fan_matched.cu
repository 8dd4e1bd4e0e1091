// Matched fan backprojection (type 2), the exact transpose of the fan forward
// projection.
//
// A view's lattice lines are image rows (X class) or columns (Y class), and a
// pixel gets half of its footprint on the two lines at its sides.  Here a lane
// owns a line of its warp's block of 31 x 31 pixels, rows or columns by the
// view's class, and steps along it: the line's distance from the source is one
// reciprocal per view, the detector's edge index a quartic of the slope, and
// the footprint of a cell of the line is the difference of the table prefixes at
// two neighbouring lattice points of the same lane.  Views are sorted by class, so
// the lines' totals turn into pixels twice in all: each pixel is its own and the
// next lane's total, and the X-class pixels wait in shared memory, transposed.
//
// With lanes along x for both classes an X-class view took two shuffles and a
// reciprocal per lattice point, and both classes their per-view terms for 17
// points instead of 32: 64 slices of 512 x 512 with 576-1152 views took 12.75 ms,
// 10.87 now.  The unrolled line wants 168 registers: 12 warps per SM are faster
// than 16 that spill (12.3 ms), and than 24 with lines of 16 cells (12.7 ms; with
// warps apart by up to three chunks instead of one barrier per chunk 14.7 ms).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "fan_bp.cuh"
#include "rn_device.cuh"
#include "rn_internal.h"

namespace rn {

constexpr int kMtBlock = 31;                   // pixels per block side: lanes 0..30, the last lane only supplies a line
constexpr int kMtWarps = 4;                    // 2 x 2 blocks
constexpr int kMtPitch = kMtBlock + 2;         // odd: rows and columns of the pixel store are free of bank conflicts
constexpr int kMtStore = kMtBlock * kMtPitch;  // floats per warp
static_assert(2 * kMtBlock == kMatchedTile, "the plan sizes windows and cubics for this tile");
constexpr int kMtSmem = 113 * 1024;            // two blocks per SM

struct MtParams {
    const ViewGeo* views;
    const GeoSet* sets;
    const BpSlice* bps;
    const float4* tab;
    long long tab_base;
    int s_begin;
    float* img;
    int* err;
    FanDims d;
    int accumulate;
    int tiles_x, tiles_y, win, nparts;
    long long spin, part_stride;
    float* parts;
};

// A view as a warp reads it: the quartic of the edge index t(r) = tA + tB
// atan(kappa r) around the slope at the middle of the warp's 31 x 31 pixels
// (ViewGeo::quartic says that it stays within 0.05 cells, usually 1e-3; it only
// selects the cell), as pairs for packed arithmetic.  Lane v works out view v of a
// chunk.
struct alignas(16) MtView {
    f32x2 c0, c1, c2, c3, c4, nrt, npar;
    float perp;
    uint32_t tbase;   // byte address of the entry of edge index 0 less the bias of the round-down add
};

// A block's shared memory with V views per staged chunk: the views' parameters,
// the pixel store, the warps' view records, then two buffers of V table windows.
// Windows widen with the pixels (in detector cells), so wide ones go with fewer
// views per chunk: as many of 8, 4 and 2 as leave room for two blocks per SM, or
// else two, which fit whatever window the plan's own limit lets through.  8 slices
// of 576 to 720 views: 256 x 256 pixels of 1.65 mm (392 entries) 0.80 ms with eight
// views (one block per SM), 0.53 with four; 128 x 128 pixels of 2.9 mm (656 entries)
// 0.35 with eight, 0.27 with four (two blocks per SM), 0.28 with two (three); 316 x
// 316 pixels of 1.2 mm (280 entries) 0.70 with eight (two blocks), 0.71 with four.
template <int V>
struct MtLayout {
    static constexpr size_t kStore = (sizeof(BpSharedT<V>) + 127) & ~size_t(127);
    static constexpr size_t kRec = (kStore + sizeof(float) * kMtWarps * kMtStore + 127) & ~size_t(127);
    static constexpr size_t kBuf = (kRec + sizeof(MtView) * kMtWarps * V + 127) & ~size_t(127);
    static size_t bytes(int win) { return kBuf + 2 * (size_t)V * win * sizeof(float4); }
};

__device__ __forceinline__ void mt_prepare(MtView& o, const BpView& vg, float lmid, float qmid, uint32_t T, int ilo) {
    const float rt = (qmid - vg.par) * __fdividef(1.0f, lmid - vg.perp), ut = vg.kappa * rt, u2 = ut * ut;
    const float iw = __fdividef(1.0f, 1.0f + u2), kw = vg.kappa * iw;
    const float c0 = fmaf(vg.tB, atanf(ut), vg.tA), c1 = vg.tB * kw, c2 = -c1 * kw * ut;
    const float c3 = c1 * kw * kw * (u2 - 1.0f / 3.0f), c4 = c1 * kw * kw * kw * ut * (1.0f - u2);
    o.c0 = f2_pack(c0, c0);
    o.c1 = f2_pack(c1, c1);
    o.c2 = f2_pack(c2, c2);
    o.c3 = f2_pack(c3, c3);
    o.c4 = f2_pack(c4, c4);
    o.nrt = f2_pack(-rt, -rt);
    o.npar = f2_pack(-vg.par, -vg.par);
    o.perp = vg.perp;
    o.tbase = T + (uint32_t)(1 - ilo - 0x4B400000) * 16u;
}

// One view: line l, lattice points q0 .. q0 + 31.  Point q's slope is (q - par)
// g; both q - par and the difference from an edge's slope are rounded once.
// kInside: the staged window holds every entry the tile can select.
template <bool kInside>
__device__ __forceinline__ void mt_view(float (&line)[kMtBlock], const MtView& vg, float l, float q0, int ilo, int imax) {
    const MtView w = vg;
    const float g = __fdividef(1.0f, l - w.perp);
    f32x2 q2 = f2_pack(q0, q0 + 1.0f);
    const f32x2 g2 = f2_pack(g, g), two2 = f2_pack(2.0f, 2.0f), bias2 = f2_pack(12582912.0f, 12582912.0f);
    float hp = 0.f, rp = 0.f;
#pragma unroll
    for (int j = 0; j <= kMtBlock; j += 2) {
        const f32x2 a2 = f2_add(q2, w.npar);
        q2 = f2_add(q2, two2);
        const f32x2 h = f2_fma(a2, g2, w.nrt);
        const f32x2 t = f2_fma(h, f2_fma(h, f2_fma(h, f2_fma(h, w.c4, w.c3), w.c2), w.c1), w.c0);
        const float2 y = f2_unpack(f2_add_rd(t, bias2)), a = f2_unpack(a2);
        int i0 = __float_as_int(y.x), i1 = __float_as_int(y.y);
        if (!kInside) {   // (biased) entries ilo .. imax
            i0 = min(max(i0, ilo + (0x4B400000 - 1)), imax + (0x4B400000 - 1));
            i1 = min(max(i1, ilo + (0x4B400000 - 1)), imax + (0x4B400000 - 1));
        }
        const float4 E0 = lds4(w.tbase + (uint32_t)i0 * 16u), E1 = lds4(w.tbase + (uint32_t)i1 * 16u);
        const float r0 = fmaf(E0.z, fmaf(a.x, g, -E0.w), E0.y), r1 = fmaf(E1.z, fmaf(a.y, g, -E1.w), E1.y);
        if (j > 0) line[j - 1] += (E0.x - hp) + (r0 - rp);
        line[j] += (E1.x - E0.x) + (r1 - r0);
        hp = E1.x;
        rp = r1;
    }
}

// The same where the quartic is not good enough (tiles near or beyond the source):
// a cubic per lane and 8 cells, clamped indices.
__device__ __forceinline__ void mt_view_near(float (&line)[kMtBlock], const BpView& vg, const float4* T, float l, float q0,
                                             int ilo, int imax) {
    const float g = __fdividef(1.0f, l - vg.perp);
    TCubic c;
    float hp = 0.f, rp = 0.f;
#pragma unroll
    for (int j = 0; j <= kMtBlock; j++) {
        if (j % 8 == 0) c = t_cubic(vg, ((q0 + (float)(j + 4)) - vg.par) * g);
        const float a = (q0 + (float)j) - vg.par, h = fmaf(a, g, -c.rt);
        const float t = fmaf(h, fmaf(h, fmaf(h, c.c3, c.c2), c.c1), c.c0);
        const float4 E = T[min(max(floor_small(t) + 1, ilo), imax) - ilo];
        const float r = fmaf(E.z, fmaf(a, g, -E.w), E.y);
        if (j > 0) line[j - 1] += (E.x - hp) + (r - rp);
        hp = E.x;
        rp = r;
    }
}

// V views per staged chunk.  kNear: some views of the plan are near ones (a
// kernel of its own: its third form of the line costs the others 4%).
template <int V, bool kNear>
__global__ void __launch_bounds__(32 * kMtWarps, 3) fan_bp_matched_kernel(MtParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    using L = MtLayout<V>;
    BpSharedT<V>* sh = reinterpret_cast<BpSharedT<V>*>(smem);
    float4* const buf0 = reinterpret_cast<float4*>(smem + L::kBuf);   // buffer b at buf0 + b * V * win

    const int tiles = p.tiles_x * p.tiles_y;
    const int part = blockIdx.x % p.nparts, bid = blockIdx.x / p.nparts;
    const int si = bid / tiles, ti = bid - si * tiles, tyi = ti / p.tiles_x, txi = ti - tyi * p.tiles_x;
    const BpSlice bs = p.bps[p.s_begin + si];
    GeoSet gs = p.sets[bs.set];
    const int nx = p.d.nx, ny = p.d.ny, tabn = p.d.nu + 2;
    const float4* gtab = p.tab + (bs.table_off - p.tab_base);
    if (p.nparts > 1) {
        // this part's share of the views, in whole chunks of the split
        const int nch = (gs.nview + kBpSplitViews - 1) / kBpSplitViews, cpp = (nch + p.nparts - 1) / p.nparts;
        const int vb = min(gs.nview, part * cpp * kBpSplitViews), ve = min(gs.nview, (part + 1) * cpp * kBpSplitViews);
        gs.view_off += vb;
        gs.nview = ve - vb;
        gtab += (long long)vb * tabn;
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int X0 = txi * kMatchedTile, Y0 = tyi * kMatchedTile;
    const int bx = X0 + (warp & 1) * kMtBlock, by = Y0 + (warp >> 1) * kMtBlock;
    const bool live = bx < nx && by < ny;   // the whole warp
    MtView* const rec = reinterpret_cast<MtView*>(smem + L::kRec) + warp * V;
    float* const store = reinterpret_cast<float*>(smem + L::kStore) + warp * kMtStore;   // pixel (bx + a, by + b) at a kMtPitch + b

    if (tid == 0) {
        mbar_init(&sh->bars[0], 1);
        mbar_init(&sh->bars[1], 1);
        fence_mbar_init();
    }
    const int nchunks = (gs.nview + V - 1) / V;
    auto prep = [&](int c, const ViewGeo* src) {
        bp_prep<V, kMatchedTile, kMatchedTile, 4>(sh, src, c, gs.nview, X0, Y0, nx, ny, tabn, p.win, 1, 2);
    };
    // tid 0: stage chunk c's table windows into buffer c & 1 and the view
    // records of chunk c + 1 into record slot (c + 1) & 1, on barrier c & 1
    auto issue = [&](int c) {
        const int b = c & 1, vc = min(V, gs.nview - c * V), cnt = min(p.win, tabn);
        const int vn = c + 1 < nchunks ? min(V, gs.nview - (c + 1) * V) : 0;
        fence_proxy_async();
        mbar_arrive_expect_tx(&sh->bars[b], (uint32_t)(vc * cnt * sizeof(float4) + vn * sizeof(ViewGeo)));
        for (int v = 0; v < vc; v++)
            bulk_g2s(buf0 + (b * V + v) * p.win, gtab + (long long)(c * V + v) * tabn + sh->elo[c % 3][v],
                     (uint32_t)(cnt * sizeof(float4)), &sh->bars[b]);
        if (vn > 0)
            bulk_g2s(sh->rec[(c + 1) & 1], p.views + gs.view_off + (c + 1) * V, (uint32_t)(vn * sizeof(ViewGeo)),
                     &sh->bars[b]);
    };
    if (nchunks > 0) {
        if (tid < 32) prep(0, p.views + gs.view_off);
        __syncthreads();
        if (tid == 0) issue(0);
    }

    float line[kMtBlock];
#pragma unroll
    for (int j = 0; j < kMtBlock; j++) line[j] = 0.f;
    const float lx = (float)(bx + lane), ly = (float)(by + lane), qx = (float)bx, qy = (float)by;
    bool xphase = true;
    // the X-class lines (row by + lane, cells along x) to pixels; row ny does not exist
    auto x_pixels = [&]() {
#pragma unroll
        for (int j = 0; j < kMtBlock; j++) {
            const float next = __shfl_down_sync(0xffffffffu, line[j], 1);
            if (lane < kMtBlock) store[j * kMtPitch + lane] = line[j] + (by + lane + 1 < ny ? next : 0.f);
            line[j] = 0.f;
        }
        __syncwarp();
    };

    // One barrier per chunk: after it every warp has finished chunk c - 1, so
    // buffer (c + 1) & 1 and record slot c & 1 may be refilled; window and
    // parameter slots rotate over three chunks because warp 0 prepares chunk
    // c + 1 while other warps may still compute chunk c - 1.
    bool ok = true;
    for (int c = 0; c < nchunks; c++) {
        const int b = c & 1;
        if (!mbar_wait(&sh->bars[b], (uint32_t)((c >> 1) & 1), p.spin)) ok = false;
        if (tid < 32 && c + 1 < nchunks) prep(c + 1, sh->rec[(c + 1) & 1]);
        if (!__syncthreads_and(ok)) {
            // chunk c's copies are the only ones in flight: wait for them
            // (bounded) before the CTA gives its shared memory back
            if (tid == 0) {
                atomicExch(p.err, RN_ERR_TIMEOUT);
                mbar_wait(&sh->bars[b], (uint32_t)((c >> 1) & 1));
            }
            ok = false;
            break;
        }
        if (tid == 0 && c + 1 < nchunks) issue(c + 1);
        if (!live) continue;
        const int slot = c % 3, vc = min(V, gs.nview - c * V), cnt = min(p.win, tabn);
        bool xv = false, in = false;
        if (lane < vc) {
            const BpView& vg = sh->vw[slot][lane];
            xv = vg.xcls != 0;
            in = vg.inside != 0;
            mt_prepare(rec[lane], vg, (float)(xv ? by : bx) + 0.5f * kMtBlock, (float)(xv ? bx : by) + 0.5f * kMtBlock,
                       smem_u32(buf0 + (b * V + lane) * p.win), sh->elo[slot][lane]);
        }
        const unsigned xmask = __ballot_sync(0xffffffffu, xv), inside = __ballot_sync(0xffffffffu, in);
        __syncwarp();
        for (int v = 0; v < vc; v++) {
            const bool xcls = (xmask >> v) & 1;
            if (xphase && !xcls) {   // once: views are sorted by class
                x_pixels();
                xphase = false;
            }
            const float l = xcls ? ly : lx, q0 = xcls ? qx : qy;
            if ((inside >> v) & 1) {
                mt_view<true>(line, rec[v], l, q0, 0, 0);
            } else {
                const int ilo = sh->elo[slot][v];
                if (kNear && !sh->vw[slot][v].good)
                    mt_view_near(line, sh->vw[slot][v], buf0 + (b * V + v) * p.win, l, q0, ilo, ilo + cnt - 1);
                else mt_view<false>(line, rec[v], l, q0, ilo, ilo + cnt - 1);   // <= nu + 1
            }
        }
        __syncwarp();   // the records are rewritten for the next chunk
    }
    if (!ok || !live) return;
    if (xphase) {
        x_pixels();
    } else {
        // the Y-class lines (column bx + lane, cells along y); column nx does not exist
#pragma unroll
        for (int j = 0; j < kMtBlock; j++) {
            const float next = __shfl_down_sync(0xffffffffu, line[j], 1);
            if (lane < kMtBlock) store[lane * kMtPitch + j] += line[j] + (bx + lane + 1 < nx ? next : 0.f);
        }
        __syncwarp();
    }
    float* out = (p.nparts > 1 ? p.parts + part * p.part_stride : p.img) + bs.img_off;
    const bool add = p.nparts == 1 && p.accumulate;
    const int y = by + lane;
    if (lane < kMtBlock && y < ny) {
        for (int a = 0; a < min(kMtBlock, nx - bx); a++) {
            float* q = out + (long long)(bx + a) * p.d.isx + (long long)y * p.d.isy;
            const float v = store[a * kMtPitch + lane];
            *q = add ? *q + v : v;
        }
    }
}

// Views per staged chunk for windows of `win` entries; 0 where not even two fit.
static int matched_views(int win) {
    if (MtLayout<8>::bytes(win) <= kMtSmem) return 8;
    if (MtLayout<4>::bytes(win) <= kMtSmem) return 4;
    return MtLayout<2>::bytes(win) <= 227 * 1024 ? 2 : 0;
}

bool fan_matched_fits(int win) { return matched_views(win) > 0; }

int fan_matched_attributes() {
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    RN_CUDA_TRY(cudaFuncSetAttribute(fan_bp_matched_kernel<8, false>, attr, kMtSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(fan_bp_matched_kernel<8, true>, attr, kMtSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(fan_bp_matched_kernel<4, false>, attr, kMtSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(fan_bp_matched_kernel<4, true>, attr, kMtSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(fan_bp_matched_kernel<2, false>, attr, 227 * 1024));
    RN_CUDA_TRY(cudaFuncSetAttribute(fan_bp_matched_kernel<2, true>, attr, 227 * 1024));
    return RN_OK;
}

// Slices s0 .. s0 + ns - 1, whose tables start at table_base, in `nparts` shares
// of the views.
int fan_matched_launch(rn_fan_plan* p, float* d_img, int accumulate, int s0, int ns, long long table_base, int nparts,
                       cudaStream_t st) {
    MtParams m;
    m.views = p->d_views_s;
    m.sets = p->d_sets;
    m.bps = p->d_bp;
    m.tab = p->d_tab;
    m.tab_base = table_base;
    m.s_begin = s0;
    m.img = d_img;
    m.err = p->d_err;
    m.d = p->dims;
    m.accumulate = accumulate;
    m.tiles_x = (p->dims.nx + kMatchedTile - 1) / kMatchedTile;
    m.tiles_y = (p->dims.ny + kMatchedTile - 1) / kMatchedTile;
    m.win = p->table_win_t;
    m.nparts = nparts;
    m.spin = p->spin_limit;
    m.part_stride = p->img_elems;
    m.parts = p->d_bp_parts;
    auto launch = [&](auto kern, size_t smem) {
        kern<<<(unsigned)(ns * m.tiles_x * m.tiles_y * nparts), 32 * kMtWarps, smem, st>>>(m);
    };
    const bool near = p->matched_near;
    switch (matched_views(m.win)) {
        case 8:
            launch(near ? fan_bp_matched_kernel<8, true> : fan_bp_matched_kernel<8, false>, MtLayout<8>::bytes(m.win));
            break;
        case 4:
            launch(near ? fan_bp_matched_kernel<4, true> : fan_bp_matched_kernel<4, false>, MtLayout<4>::bytes(m.win));
            break;
        default:
            launch(near ? fan_bp_matched_kernel<2, true> : fan_bp_matched_kernel<2, false>, MtLayout<2>::bytes(m.win));
    }
    RN_CUDA_TRY(cudaGetLastError());
    return RN_OK;
}

}  // namespace rn
