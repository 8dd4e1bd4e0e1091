// Fan backprojection of several slices that share their views (the reference
// layout: batches, image planes and channels of one angle list), reference mode
// (typeProjector 0 / 1) and pixel driven.
//
// fan.cu's kernels work out a pixel's detector coordinates for every slice
// again: about 30 of their 40 instructions per pixel and view.  Here a block
// takes four or eight slices at once.  The per-view table holds the slices'
// sinogram values side by side (one float4 per detector cell), a pixel's cells
// and their weights are worked out once, and each slice adds a few packed
// multiply-adds:
//   reference mode: the mean of the pre-weighted sinogram over the interval
//     between the detector coordinates of the pixel's two edges, as the K cells
//     it can touch, each weighted by its overlap (the quantity that fan.cu's
//     reference mode takes from the detector prefix);
//   pixel driven: the two cells around the ray through the pixel centre
//     (pd_sample in fan.cu has the derivation).
// Tiles are 32 columns (31 in reference mode, whose last lane only supplies an
// edge) x 64 rows, or 32 rows with eight slices: a warp's lanes are the columns, a
// lane holds 16 or 8 rows of every slice.
//
// Measured: 16 slices of 512 x 512, 701 views of 888 channels, pixel driven: 5.62
// ms with fan.cu's kernel, 2.18 ms with four slices per block, 1.71 with eight
// (tables 0.11 and 0.04 ms); 12 slices of 301 x 333, 413 views of 611 channels,
// reference mode: 0.93, 0.52 and 0.53 ms (three quads fill two blocks of two by
// three quarters).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "fan_bp.cuh"
#include "rn_device.cuh"
#include "rn_internal.h"

namespace rn {

constexpr int kBgSlices = 4;    // slices per table entry (a quad); a block takes one or two quads
constexpr int kBgViews = 4;     // views per staged chunk
constexpr int kBgWarps = 4;
__host__ __device__ constexpr int bg_rows(int quads) { return 16 / quads; }   // rows per lane
__host__ __device__ constexpr int bg_tile_y(int quads) { return kBgWarps * bg_rows(quads); }
constexpr int kBgPad = 4;       // zero cells on both sides of a table row: cell u at entry u + kBgPad
constexpr int kBgSmem = 100 * 1024;   // at least two blocks per SM
using BgShared = BpSharedT<kBgViews>;

struct GroupParams {
    const ViewGeo* views;
    const BpSlice* bps;
    const float4* vals;     // [group][view][tabn]
    const float2* geo;      // [view][tabn] (pixel driven): slope of the ray through the cell's centre, hi / lo
    float* img;
    int* err;
    FanDims d;
    int s_begin, ns, view_off, nview, tabn, win;
    int accumulate, fbp;
    int tiles_x, tiles_y, nparts;
    long long spin, part_stride;
    float* parts;
};

// Values of kBgSlices slices (mixed over their detector rows; with the length
// weight of fan_table_kernel when `len`), and the slopes of the cells' rays
// when `geo` is given.  32 views x 32 cells per block through shared memory, so
// that the sinogram is read along its views and the table written along its
// cells.  Block (32, 8): blockIdx = (view tile, cell tile, group).
__global__ void __launch_bounds__(256) fan_group_table_kernel(float4* __restrict__ vals, float2* __restrict__ geo,
                                                              const float* __restrict__ prj,
                                                              const BpSlice* __restrict__ bps, int s_begin, int ns,
                                                              const ViewGeo* __restrict__ views,
                                                              const double* __restrict__ cslopes,
                                                              const float2* __restrict__ cell, FanDims d, int nview,
                                                              int tabn, int len) {
    __shared__ float tile[kBgSlices][32][33];
    const int lane = threadIdx.x, w = threadIdx.y;
    const int v0 = blockIdx.x * 32, i0 = blockIdx.y * 32, g = blockIdx.z;
    const int nu = d.nu;
    const int view = v0 + lane;
#pragma unroll
    for (int s = 0; s < kBgSlices; s++) {
        const int si = g * kBgSlices + s;
        const bool have = si < ns && view < nview;
        const BpSlice bs = bps[s_begin + min(si, ns - 1)];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int u = i0 + w + 8 * k - kBgPad;
            float val = 0.f;
            if (have && (unsigned)u < (unsigned)nu) {
#pragma unroll
                for (int j = 0; j < kBpMix; j++) {
                    const float wj = bs.prj_w[j];
                    if (wj != 0.f)
                        val += wj * __ldg(prj + bs.prj_off[j] + (long long)u * bs.su + (long long)view * bs.sview);
                }
                if (len) {
                    const ViewGeo& vg = views[view];
                    const float2 cs = cell[u];
                    val *= vg.xcls ? d.dy / fabsf(vg.cosd * cs.x + vg.sind * cs.y)
                                   : d.dx / fabsf(vg.sind * cs.x - vg.cosd * cs.y);
                }
            }
            tile[s][w + 8 * k][lane] = val;
        }
    }
    __syncthreads();
    const int idx = i0 + lane;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int vw = w + 8 * k, v = v0 + vw;
        if (v < nview && idx < tabn)
            vals[((long long)g * nview + v) * tabn + idx] =
                make_float4(tile[0][lane][vw], tile[1][lane][vw], tile[2][lane][vw], tile[3][lane][vw]);
    }
    if (geo && g == 0) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int v = v0 + w + 8 * k, u = idx - kBgPad;
            if (v >= nview || idx >= tabn) continue;
            double r = 0.0;
            const double* row = cslopes + (long long)v * (nu + 1);
            if (u >= 0 && u <= nu) {
                r = row[u];
            } else if (u == -1) {   // the ray one cell pitch before the first (pd_table_kernel)
                const int xcls = views[v].xcls;
                const double kap = xcls ? (double)d.dx / d.dy : (double)d.dy / d.dx;
                const double rho = kap * row[0], tn = tan((double)d.du);
                r = (xcls ? (rho + tn) / (1.0 - rho * tn) : (rho - tn) / (1.0 + rho * tn)) / kap;
            }
            const float rh = (float)r;
            geo[(long long)v * tabn + idx] = make_float2(rh, (float)(r - (double)rh));
        }
    }
}

__device__ __forceinline__ f32x2 f2_dup(float v) { return f2_pack(v, v); }

// acc += scale sum_k w[k] T[i + k], the four slices of each entry in two pairs; the
// second quad's window is `win` entries on.  The cells are added up before they join
// the views' running sums, each of whose roundings weighs as much as all of a view's:
// in reference mode 360 views of 1 mm pixels are 8.7e-8 off so and 9.1e-8 with every
// cell added to the running sum, 900 views 9.4e-8 and 1.2e-7 (relative L2).
template <int K, int Q>
__device__ __forceinline__ void add_cells(f32x2 (&acc)[2 * Q], const float4* T, int win, const float (&w)[K], float scale) {
    f32x2 t[2 * Q];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const f32x2 ww = f2_dup(w[k]);
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const ulonglong2 E = *reinterpret_cast<const ulonglong2*>(T + k + q * win);
            t[2 * q] = k ? f2_fma(ww, E.x, t[2 * q]) : f2_mul(ww, E.x);
            t[2 * q + 1] = k ? f2_fma(ww, E.y, t[2 * q + 1]) : f2_mul(ww, E.y);
        }
    }
#pragma unroll
    for (int q = 0; q < 2 * Q; q++) acc[q] = f2_fma(f2_dup(scale), t[q], acc[q]);
}

// Reference mode: the K cells under the interval between the detector coordinates
// t0, t1 (cell edges at integers), each by its overlap, times `scale` over its width.
template <int K, int Q>
__device__ __forceinline__ void add_interval(f32x2 (&acc)[2 * Q], const float4* T, int win, int ilo, int imax, float t0,
                                             float t1, float scale) {
    const float lo = fminf(t0, t1), width = fabsf(t1 - t0);
    const float y = __fadd_rd(lo, 12582912.0f);
    const float f = lo - (y - 12582912.0f);
    int i = __float_as_int(y) - 0x4B400000 + kBgPad;
    i = min(max(i, ilo), imax - (K - 1));   // off the detector: zero cells
    const float iw = __fdividef(scale, width);
    float w[K], rest = width, o = fminf(1.0f - f, rest);
    w[0] = o;
#pragma unroll
    for (int k = 1; k < K - 1; k++) {
        rest -= o;
        o = fminf(1.0f, rest);
        w[k] = o;
    }
    w[K - 1] = rest - o;
    add_cells<K, Q>(acc, T + (i - ilo), win, w, iw);
}

// kMode 0: reference mode with K cells; 3: pixel driven (K = 2).  Q quads of
// slices.
template <int kMode, int K, int Q>
__global__ void __launch_bounds__(32 * kBgWarps, 3) fan_bp_group_kernel(GroupParams p) {
    constexpr int kCols = kMode == 3 ? 32 : 31, kRows = bg_rows(Q), kTileY = bg_tile_y(Q);
    extern __shared__ __align__(128) unsigned char smem[];
    BgShared* sh = reinterpret_cast<BgShared*>(smem);
    const size_t off = (sizeof(BgShared) + 127) & ~size_t(127);
    float4* const buf0 = reinterpret_cast<float4*>(smem + off);                   // [2][kBgViews][Q][win]
    float2* const geo0 = reinterpret_cast<float2*>(buf0 + 2 * kBgViews * Q * p.win);   // [2][kBgViews][win]
    const int tiles = p.tiles_x * p.tiles_y;
    const int part = blockIdx.x % p.nparts, bid = blockIdx.x / p.nparts;
    const int grp = bid / tiles, ti = bid - grp * tiles;
    const int tyi = ti / p.tiles_x, txi = ti - tyi * p.tiles_x;
    // this part's share of the views, in whole chunks
    const int nch_all = (p.nview + kBgViews - 1) / kBgViews, cpp = (nch_all + p.nparts - 1) / p.nparts;
    const int vbeg = min(p.nview, part * cpp * kBgViews), nview = min(p.nview, (part + 1) * cpp * kBgViews) - vbeg;
    const ViewGeo* views = p.views + p.view_off + vbeg;
    // the block's first quad, and the distance to the second (0 where there is none: staged again, not stored)
    const float4* gval = p.vals + ((long long)grp * Q * p.nview + vbeg) * p.tabn;
    const long long second = grp * Q + 1 < (p.ns + kBgSlices - 1) / kBgSlices ? (long long)p.nview * p.tabn : 0;
    const float2* ggeo = p.geo + (long long)vbeg * p.tabn;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int X0 = txi * kCols, Y0 = tyi * kTileY;
    const int x0 = X0 + lane, y0 = Y0 + warp * kRows;
    const int win = p.win;   // even, and at most tabn, so that every window starts on an even entry
    if (tid == 0) {
        mbar_init(&sh->bars[0], 1);
        mbar_init(&sh->bars[1], 1);
        fence_mbar_init();
    }
    const int nchunks = (nview + kBgViews - 1) / kBgViews;
    auto prep = [&](int c, const ViewGeo* src) {
        bp_prep<kBgViews, kCols, kTileY>(sh, src, c, nview, X0, Y0, p.d.nx, p.d.ny, p.tabn, win, kBgPad, 3);
    };
    auto issue = [&](int c) {
        const int b = c & 1;
        const int vc = min(kBgViews, nview - c * kBgViews);
        const int vn = c + 1 < nchunks ? min(kBgViews, nview - (c + 1) * kBgViews) : 0;
        const uint32_t entry = Q * sizeof(float4) + (kMode == 3 ? sizeof(float2) : 0);
        fence_proxy_async();
        mbar_arrive_expect_tx(&sh->bars[b], (uint32_t)(vc * win * entry + vn * sizeof(ViewGeo)));
        for (int v = 0; v < vc; v++) {
            const long long row = (long long)(c * kBgViews + v) * p.tabn + (sh->elo[c % 3][v] & ~1);
#pragma unroll
            for (int q = 0; q < Q; q++)
                bulk_g2s(buf0 + ((b * kBgViews + v) * Q + q) * win, gval + q * second + row,
                         (uint32_t)(win * sizeof(float4)), &sh->bars[b]);
            if (kMode == 3)
                bulk_g2s(geo0 + (b * kBgViews + v) * win, ggeo + row, (uint32_t)(win * sizeof(float2)), &sh->bars[b]);
        }
        if (vn > 0)
            bulk_g2s(sh->rec[(c + 1) & 1], views + (c + 1) * kBgViews, (uint32_t)(vn * sizeof(ViewGeo)), &sh->bars[b]);
    };
    if (nchunks > 0) {
        if (tid < 32) prep(0, views);
        __syncthreads();
        if (tid == 0) issue(0);
    }
    f32x2 acc[kRows][2 * Q];
#pragma unroll
    for (int j = 0; j < kRows; j++)
#pragma unroll
        for (int q = 0; q < 2 * Q; q++) acc[j][q] = 0ull;
    const float dso2 = p.d.dso * p.d.dso;
    // one barrier per chunk, as in fan_bp_kernel
    bool ok = true;
    for (int c = 0; c < nchunks; c++) {
        const int b = c & 1;
        if (!mbar_wait(&sh->bars[b], (uint32_t)((c >> 1) & 1), p.spin)) ok = false;
        if (tid < 32 && c + 1 < nchunks) prep(c + 1, sh->rec[(c + 1) & 1]);
        if (!__syncthreads_and(ok)) {
            // chunk c's copies are the only ones in flight: wait for them
            // (bounded) before the block gives its shared memory back
            if (tid == 0) {
                atomicExch(p.err, RN_ERR_TIMEOUT);
                mbar_wait(&sh->bars[b], (uint32_t)((c >> 1) & 1));
            }
            ok = false;
            break;
        }
        if (tid == 0 && c + 1 < nchunks) issue(c + 1);
        const int slot = c % 3, vc = min(kBgViews, nview - c * kBgViews);
        for (int v = 0; v < vc; v++) {
            const BpView vg = sh->vw[slot][v];
            const float4* T = buf0 + (b * kBgViews + v) * Q * win;
            const float2* G = geo0 + (b * kBgViews + v) * win;
            const int ilo = sh->elo[slot][v] & ~1, imax = ilo + win - 1;
            const bool xc = vg.xcls;
            const float dq = xc ? p.d.dx : p.d.dy, dl = xc ? p.d.dy : p.d.dx;
            if (kMode == 0) {
                if (xc) {
                    const float A = (float)x0 - vg.par, aq = (A + 0.5f) * dq;
                    const TCubic cu = t_cubic(vg, A * __fdividef(1.0f, (float)(y0 + kRows / 2) - vg.perp));
#pragma unroll
                    for (int j = 0; j < kRows; j++) {
                        const float D = (float)(y0 + j) + 0.5f - vg.perp;
                        const float h = A * __fdividef(1.0f, D) - cu.rt;
                        const float t = fmaf(h, fmaf(h, fmaf(h, cu.c3, cu.c2), cu.c1), cu.c0);
                        const float nt = __shfl_down_sync(0xffffffffu, t, 1);
                        const float bl = D * dl;
                        add_interval<K, Q>(acc[j], T, win, ilo, imax, t, nt,
                                        p.fbp ? __fdividef(dso2, fmaf(aq, aq, bl * bl)) : 1.0f);
                    }
                } else {
                    const float D = (float)x0 + 0.5f - vg.perp, g = __fdividef(1.0f, D), bl = D * dl;
                    const float r0 = ((float)y0 - vg.par) * g;
                    const TCubic cu = t_cubic(vg, fmaf((float)(kRows / 2), g, r0));
                    float tp = 0.f;
#pragma unroll
                    for (int j = 0; j <= kRows; j++) {
                        const float h = fmaf((float)j, g, r0) - cu.rt;
                        const float t = fmaf(h, fmaf(h, fmaf(h, cu.c3, cu.c2), cu.c1), cu.c0);
                        if (j > 0) {
                            const float a = ((float)(y0 + j) - 0.5f - vg.par) * dq;
                            add_interval<K, Q>(acc[j - 1], T, win, ilo, imax, tp, t,
                                            p.fbp ? __fdividef(dso2, fmaf(a, a, bl * bl)) : 1.0f);
                        }
                        tp = t;
                    }
                }
            } else {
                // pixel driven: offsets from the source along (A) and across
                // (D) the lines as hi / lo floats
                float Ah, Al, Dh, Dl;
                const float q0 = xc ? (float)x0 : (float)y0, l0 = xc ? (float)y0 : (float)x0;
                split_hilo(vg.pard - ((double)q0 + 0.5), Ah, Al);
                split_hilo(((double)l0 + 0.5) - vg.perpd, Dh, Dl);
                const float A = q0 + 0.5f - vg.par, g = __fdividef(1.0f, l0 + 0.5f - vg.perp);
                const TCubic cu = t_cubic(vg, xc ? A * __fdividef(1.0f, l0 + (float)(kRows / 2) - vg.perp)
                                                 : fmaf((float)(kRows / 2) - 0.5f, g, A * g));
                const float cfrac = -vg.tB * dq * dl;
#pragma unroll
                for (int j = 0; j < kRows; j++) {
                    float a_h = Ah, a_l = Al, d_h = Dh, d_l = Dl, e, r;
                    if (xc) {
                        r = A * __fdividef(1.0f, l0 + (float)j + 0.5f - vg.perp);
                        two_sum(Dh, (float)j, d_h, e);
                        d_l = Dl + e;
                    } else {
                        r = fmaf((float)j, g, A * g);
                        two_sum(Ah, -(float)j, a_h, e);
                        a_l = Al + e;
                    }
                    const float h = r - cu.rt;
                    const float t = fmaf(h, fmaf(h, fmaf(h, cu.c3, cu.c2), cu.c1), cu.c0);
                    int i = floor_small(t - 0.5f) + kBgPad;
                    i = min(max(i, ilo), imax - 1);
                    const float2 R = G[i - ilo];
                    const float xu = fmaf(R.x, d_h, a_h) + fmaf(R.y, d_h, fmaf(R.x, d_l, a_l));
                    const float a = a_h * dq, bl = d_h * dl;
                    const float il2 = __fdividef(1.0f, fmaf(a, a, bl * bl));
                    const float xl = xu * il2;
                    const float frac = cfrac * d_h * xl * fmaf(dq * a, xl, 1.0f);
                    // before the centre of the first cell's zero neighbour: nothing
                    const float wgt = (i < kBgPad && frac < 0.f) ? 0.f : dso2 * il2;
                    const float w[2] = {1.0f - frac, frac};
                    add_cells<2, Q>(acc[j], T + (i - ilo), win, w, wgt);
                }
            }
        }
    }
    if (!ok) return;
    if (lane < kCols && x0 < p.d.nx) {
        float* base = p.nparts > 1 ? p.parts + part * p.part_stride : p.img;
        const bool add = p.nparts == 1 && p.accumulate;
#pragma unroll
        for (int s = 0; s < Q * kBgSlices; s++) {
            const int si = grp * Q * kBgSlices + s;
            if (si >= p.ns) break;
            float* out = base + p.bps[p.s_begin + si].img_off + (long long)x0 * p.d.isx;
#pragma unroll
            for (int j = 0; j < kRows; j++) {
                const int iy = y0 + j;
                if (iy < p.d.ny) {
                    const float2 a = f2_unpack(acc[j][s / 2]);
                    const float v = s & 1 ? a.y : a.x;
                    float* q = out + (long long)iy * p.d.isy;
                    *q = add ? *q + v : v;
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
static int group_tabn(const rn_fan_plan* p) { return (p->dims.nu + 2 * kBgPad + 1) & ~1; }

// Staged entries per view: the detector extent of a tile at the point
// closest to the source, with the cells before and after it; 0 where the
// window does not fit.
static int group_window(const rn_fan_plan* p, int quads) {
    const RnFanGeom& g = p->g;
    const double tw = 32 * (double)g.dx, th = bg_tile_y(quads) * (double)g.dy;
    const double hx = g.nx * (double)g.dx / 2 + std::fabs(g.cx), hy = g.ny * (double)g.dy / 2 + std::fabs(g.cy);
    const double dmin = g.dso - std::sqrt(hx * hx + hy * hy);
    if (!(dmin > 0)) return 0;
    const double w = std::sqrt(tw * tw + th * th) / (dmin * g.du) + 14;
    if (!(w < 4096)) return 0;
    return std::min(((int)std::ceil(w) + 7) & ~7, group_tabn(p));
}

static size_t group_smem(int win, int quads) {
    return ((sizeof(BgShared) + 127) & ~size_t(127)) +
           2 * (size_t)kBgViews * win * (quads * sizeof(float4) + sizeof(float2));
}

// Quads per block: two (a pixel's cells and weights cost about 45 instructions, a
// quad about 8) where their windows fit and the quads fill the blocks, or nearly:
// 12 slices in two blocks of two quads take as long as in three of one.
static int group_quads(const rn_fan_plan* p, int ns) {
    const int win = group_window(p, 2);
    const int groups = (ns + kBgSlices - 1) / kBgSlices;
    return (groups % 2 == 0 || groups >= 5) && win >= 8 && group_smem(win, 2) <= (size_t)kBgSmem ? 2 : 1;
}

// Most cells a pixel's interval can span in reference mode.
static double group_width(const rn_fan_plan* p) {
    const RnFanGeom& g = p->g;
    const double hx = g.nx * (double)g.dx / 2 + std::fabs(g.cx), hy = g.ny * (double)g.dy / 2 + std::fabs(g.cy);
    return std::max(g.dx, g.dy) / ((g.dso - std::sqrt(hx * hx + hy * hy)) * g.du);
}

// The grouped kernels take a launch of `ns` slices where sharing the geometry
// pays (three slices or more: two gain little over fan.cu's kernels and leave
// half of a group empty), the table scratch holds the groups' tables, and a
// pixel spans at most 3 cells (reference mode).
bool fan_group_ok(const rn_fan_plan* p, int type, int ns) {
    if (p->ragged || ns < 3) return false;
    if (type != RN_TYPE_ITERATIVE && type != RN_TYPE_FBP && type != RN_TYPE_PIXEL) return false;
    const int win = group_window(p, 1);
    if (win < 8 || group_smem(win, 1) > (size_t)kBgSmem) return false;
    if (type != RN_TYPE_PIXEL && !(group_width(p) <= 2.99)) return false;
    const long long rows = (long long)p->total_views * group_tabn(p);
    const long long groups = (ns + kBgSlices - 1) / kBgSlices;
    return groups * rows + (type == RN_TYPE_PIXEL ? (rows + 1) / 2 : 0) <= p->tab_elems;
}

int fan_group_attributes() {
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    RN_CUDA_TRY(cudaFuncSetAttribute(fan_bp_group_kernel<0, 3, 1>, attr, kBgSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(fan_bp_group_kernel<0, 3, 2>, attr, kBgSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(fan_bp_group_kernel<0, 4, 1>, attr, kBgSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(fan_bp_group_kernel<0, 4, 2>, attr, kBgSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(fan_bp_group_kernel<3, 2, 1>, attr, kBgSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(fan_bp_group_kernel<3, 2, 2>, attr, kBgSmem));
    return RN_OK;
}

int fan_group_backproject(rn_fan_plan* p, float* d_img, const float* d_prj, int type, int accumulate, int s0, int ns,
                          int* nparts, cudaStream_t st) {
    const FanDims& d = p->dims;
    const int quads = group_quads(p, ns), nview = (int)p->total_views, tabn = group_tabn(p), win = group_window(p, quads);
    const bool pixel = type == RN_TYPE_PIXEL;
    const int groups = (ns + kBgSlices - 1) / kBgSlices;
    float4* vals = p->d_tab;
    float2* geo = pixel ? reinterpret_cast<float2*>(p->d_tab + (long long)groups * nview * tabn) : nullptr;
    {
        LaunchScope ls(p, st, 2);
        fan_group_table_kernel<<<dim3((nview + 31) / 32, (tabn + 31) / 32, groups), dim3(32, 8), 0, st>>>(
            vals, geo, d_prj, p->d_bpr, s0, ns, p->d_views, p->d_cslopes, p->d_cell, d, nview, tabn,
            type == RN_TYPE_ITERATIVE ? 1 : 0);
    }
    RN_CUDA_TRY(cudaGetLastError());
    GroupParams g;
    g.views = p->d_views;
    g.bps = p->d_bpr;
    g.vals = vals;
    g.geo = geo ? geo : reinterpret_cast<const float2*>(vals);
    g.img = d_img;
    g.err = p->d_err;
    g.d = d;
    g.s_begin = s0;
    g.ns = ns;
    g.view_off = 0;
    g.nview = nview;
    g.tabn = tabn;
    g.win = win;
    g.accumulate = accumulate;
    g.fbp = type == RN_TYPE_FBP;
    const int cols = pixel ? 32 : 31;
    g.tiles_x = (d.nx + cols - 1) / cols;
    g.tiles_y = (d.ny + bg_tile_y(quads) - 1) / bg_tile_y(quads);
    g.spin = p->spin_limit;
    // too few blocks to fill the GPU: split each tile's views (tuned, or
    // towards six blocks per SM), as far as the plan's scratch goes
    const long long ctas = (long long)g.tiles_x * g.tiles_y * ((groups + quads - 1) / quads);
    const int nch = (nview + kBgViews - 1) / kBgViews;
    long long want = 1;
    if (ns == (int)p->h_bpr.size() && p->bp_parts_cap > 0) {
        want = p->bp_nparts > 0 ? p->bp_nparts : (6LL * 148 + ctas - 1) / ctas;
        want = std::min<long long>(std::min<long long>(want, kBpMaxParts), std::min<long long>(nch, p->bp_parts_cap / p->img_elems));
    }
    g.nparts = (int)std::max<long long>(want, 1);
    g.part_stride = p->img_elems;
    g.parts = p->d_bp_parts;
    *nparts = g.nparts;
    const unsigned grid = (unsigned)(ctas * g.nparts);
    const size_t smem = group_smem(win, quads);
    LaunchScope ls(p, st, 3);
    auto launch = [&](auto kern) { kern<<<grid, 32 * kBgWarps, smem, st>>>(g); };
    if (pixel) quads == 2 ? launch(fan_bp_group_kernel<3, 2, 2>) : launch(fan_bp_group_kernel<3, 2, 1>);
    else if (group_width(p) <= 1.99) quads == 2 ? launch(fan_bp_group_kernel<0, 3, 2>) : launch(fan_bp_group_kernel<0, 3, 1>);
    else quads == 2 ? launch(fan_bp_group_kernel<0, 4, 2>) : launch(fan_bp_group_kernel<0, 4, 1>);
    RN_CUDA_TRY(cudaGetLastError());
    return RN_OK;
}

}  // namespace rn
