// Siddon cone-beam pair for tomosynthesis: a detector perpendicular to the z
// axis with u along x and v along y, every view's main axis z.  A ray's x
// depends on iu only and its y on iv only, so in a unit slab along z ray (iu,
// iv) meets at most one x grid line, at a time ta(iu), and one y grid line, at
// tb(iv), and everything but the values is worked out per iu and per iv of a
// tile instead of per ray or voxel and view.  Values come from a patch staged
// in shared memory.
//
// Forward projection (cone_fp_tile_kernel): a block owns a tile of rays of one
// view and steps through the slabs; a lane keeps the voxels j0, j1 and the time
// tb of its rows iv, and a warp walks its columns iu with the values of the two
// voxel rows a column can touch.  A column that stays in one voxel row adds tb
// I(j0) + (1 - tb) I(j1); one that crosses splits both shares at ta.
//
// Backprojection (cone_bp_tile_kernel), the exact transpose as a gather: a block
// owns a tile of voxels and walks the views; a lane keeps the few rows iv that
// can meet its voxel, with the part of the slab each spends inside its y range;
// a warp walks the columns iu in the order of the voxels they meet.  A column
// that stays in one voxel adds the sum over the lane's rows of value x time; one
// that crosses gives its first part [0, ta] to the voxel it leaves and the rest
// to the next.
//
// Positions are 64-bit fixed point (2^-32 or 2^-40 voxels).
//
// Measured, 512x512x128 voxels, 736x736 cells, 25 views: forward 1.70 ms with
// the plane-major copy (3.98 ms for cone_fp_staged_kernel, one thread per ray),
// back 3.00 ms with the weighting (6.42 ms for cone_bp_sep_kernel, which works
// out each lane's rows once per voxel pair).  Both are bound by instruction
// issue.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "cone_internal.h"
#include "rn_device.cuh"
#include "rn_internal.h"

namespace rn {

constexpr double kTileNarrow = 0.95, kTileWide = 1.9;   // widest ray spacing, in voxels, of the two FP tiles
constexpr int kFpTileSmem = 70 * 1024;                  // with the static tables, three blocks per SM
constexpr int kBpTileSmem = 69 * 1024;                  // three blocks per SM, or two for wide patches
constexpr int kBpTileSmemWide = 108 * 1024;

// Plane-major copy of one (b, c) volume, vol[z][x][pitch], y fastest, pitch =
// ny rounded up to 4, the padding zero.  32 x 32 (y, z) tiles through shared
// memory.  Block (32, 8): blockIdx = (y tile, z tile, x strip).
__global__ void __launch_bounds__(256) cone_planes_kernel(float* __restrict__ vol, const float* __restrict__ img,
                                                          ConeDims cd, int pitch, int bt, int c) {
    __shared__ float tile[32][33];
    const int y0 = blockIdx.x * 32, z0 = blockIdx.y * 32;
    const int lane = threadIdx.x, w = threadIdx.y;
    const int nx = cd.n[0], ny = cd.n[1], nz = cd.n[2];
    for (int x = blockIdx.z; x < nx; x += gridDim.z) {
        const float* base = img + bt * cd.img_b + (long long)x * cd.st[0] + c;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int y = y0 + w + 8 * k, z = z0 + lane;
            tile[w + 8 * k][lane] = (y < ny && z < nz) ? base[(long long)y * cd.st[1] + (long long)z * cd.nc] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int z = z0 + w + 8 * k, y = y0 + lane;
            if (z < nz && y < pitch) vol[((long long)z * nx + x) * pitch + y] = tile[lane][w + 8 * k];
        }
        __syncthreads();
    }
}

// Time of the grid-line crossing of a ray that moves by `step` from position
// p in one slab (ir = |1 / step|), 1 where it crosses none.
__device__ __forceinline__ float cross_time(long long p, long long step, float ir) {
    const float f = __uint2float_rn((unsigned)p) * 2.3283064365386963e-10f;
    const bool moved = (int)((p + step) >> 32) != (int)(p >> 32);
    return moved ? fminf((step > 0 ? 1.f - f : f) * ir, 1.f) : 1.f;
}

// UPW columns and 64 NP rows per warp, 4 warps along u; A the most voxel rows by
// which neighbouring columns can lie apart (ray spacing at most A - 0.1).
template <int A, int UPW, int NP>
__global__ void __launch_bounds__(128, 3) cone_fp_tile_kernel(float* __restrict__ prj, const float* __restrict__ vol,
                                                               const TileView* __restrict__ views, ConeDims cd,
                                                               int pitch, int bt, int c) {
    constexpr int TU = 4 * UPW, TV = 64 * NP;
    extern __shared__ __align__(16) float smem[];
    __shared__ float2 s_ta[4][UPW];   // crossing times, twice (both halves of a pair)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nx = cd.n[0], nz = cd.n[2];
    const int view = blockIdx.z;
    const int u0 = blockIdx.y * TU, v0 = blockIdx.x * TV, uw = u0 + warp * UPW;
    const TileView V = views[view];
    const int prows = min((int)(TU * kTileWide) + 4, (int)(TU * V.gu_max) + 4);
    const int pcols = ((int)(TV * V.gv_max) + 4 + 6) & ~3;
    const int patch = prows * pcols;
    const int S = min(4, kFpTileSmem / (4 * patch));   // >= 2 (the host's limit on the spacing)
    auto pos = [](double s, double r, double sm) { return to_fixed(fma(-sm, r, s)); };   // at slab 0
    const double ru0 = fma((double)u0, V.ru1, V.ru0), rv0 = fma((double)v0, V.rv1, V.rv0);
    const long long pu0 = pos(V.su, ru0, V.sm), du0 = to_fixed(ru0), pv0 = pos(V.sv, rv0, V.sm), dv0 = to_fixed(rv0);
    const double ru = fma((double)(uw + lane % UPW), V.ru1, V.ru0);
    long long pu = pos(V.su, ru, V.sm);
    const long long du = to_fixed(ru);
    const float iru = fabs(ru) > 1e-30 ? (float)(1.0 / fabs(ru)) : 1e30f;
    long long pv[2 * NP], dv[2 * NP];
    float irv[2 * NP];
#pragma unroll
    for (int q = 0; q < 2 * NP; q++) {
        const double rv = fma((double)(v0 + lane + 32 * q), V.rv1, V.rv0);
        pv[q] = pos(V.sv, rv, V.sm);
        dv[q] = to_fixed(rv);
        irv[q] = fabs(rv) > 1e-30 ? (float)(1.0 / fabs(rv)) : 1e30f;
    }
    // first patch row and column (a multiple of 4) of a slab: the lower of the
    // tile's first ray's two ends
    auto low = [](long long p, long long step) { return min((int)(p >> 32), (int)((p + step) >> 32)); };
    auto issue = [&](int k, int slot) {
        const int ib = low(pu0 + k * du0, du0), jb = low(pv0 + k * dv0, dv0) & ~3;
        const int j = jb + 4 * lane;
        const float* row = vol + ((long long)k * nx + ib + warp) * pitch + j;
        const uint32_t dst = smem_u32(smem + slot * patch) + (warp * pcols + 4 * lane) * 4;
        for (int q = 0; q < pcols; q += 128) {
            if (4 * lane + q >= pcols) break;
            const bool jin = j + q >= 0 && j + q < pitch;
            const float* s = row + q;
            uint32_t t = dst + 4 * q;
#pragma unroll 4
            for (int r = warp; r < prows; r += 4) {
                const bool in = jin && (unsigned)(ib + r) < (unsigned)nx;
                cp_async16(t, in ? s : vol, in);
                s += 4 * pitch;
                t += 16 * pcols;
            }
        }
    };
    f32x2 acc[UPW][NP];
#pragma unroll
    for (int k = 0; k < UPW; k++)
#pragma unroll
        for (int q = 0; q < NP; q++) acc[k][q] = 0ull;
    for (int s = 0; s < S - 1; s++) {
        if (s < nz) issue(s, s);
        cp_async_commit();
    }
    const f32x2 one = f2_pack(1.f, 1.f), minus = f2_pack(-1.f, -1.f);
    int slot = 0, fill = S - 1;
    for (int k = 0; k < nz; k++) {
        if (S == 2) cp_async_wait<0>();
        else if (S == 3) cp_async_wait<1>();
        else cp_async_wait<2>();
        __syncthreads();   // slab k is in; every warp has left the slot filled next
        if (k + S - 1 < nz) issue(k + S - 1, fill);
        cp_async_commit();
        const int now = slot;
        slot = slot + 1 == S ? 0 : slot + 1;
        fill = fill + 1 == S ? 0 : fill + 1;
        if (uw >= cd.nu) continue;   // the whole warp: columns beyond the detector
        const int ib = low(pu0 + k * du0, du0), jb = low(pv0 + k * dv0, dv0) & ~3;
        const float ta = cross_time(pu, du, iru);
        if (lane < UPW) s_ta[warp][lane] = make_float2(ta, ta);
        const int c0 = (int)(pu >> 32), c1 = (int)((pu + du) >> 32);
        const int row = min(c0, c1) - ib;
        const int before = __shfl_up_sync(0xffffffffu, row, 1);
        const unsigned adv1 = __ballot_sync(0xffffffffu, row > before);
        const unsigned adv2 = A > 1 ? __ballot_sync(0xffffffffu, row > before + 1) : 0u;
        const unsigned crosses = __ballot_sync(0xffffffffu, c0 != c1), down = __ballot_sync(0xffffffffu, c1 < c0);
        const int first = __shfl_sync(0xffffffffu, row, 0);
        const float* next[2 * NP][2];   // next patch row at this lane's voxels j0 and j1
        f32x2 tb[NP], nb[NP];           // tb and 1 - tb
        float tbs[2 * NP];
#pragma unroll
        for (int q = 0; q < 2 * NP; q++) {
            const float* base = smem + now * patch + first * pcols - jb;
            next[q][0] = base + (int)(pv[q] >> 32);
            next[q][1] = base + (int)((pv[q] + dv[q]) >> 32);
            tbs[q] = cross_time(pv[q], dv[q], irv[q]);
        }
#pragma unroll
        for (int q = 0; q < NP; q++) {
            tb[q] = f2_pack(tbs[2 * q], tbs[2 * q + 1]);
            nb[q] = f2_fma(minus, tb[q], one);
        }
        f32x2 Ra[2][NP], Rb[2][NP];   // the two rows' values at j0 and at j1
        auto load = [&](int s) {
#pragma unroll
            for (int q = 0; q < NP; q++) {
                Ra[s][q] = f2_pack(*next[2 * q][0], *next[2 * q + 1][0]);
                Rb[s][q] = f2_pack(*next[2 * q][1], *next[2 * q + 1][1]);
            }
#pragma unroll
            for (int q = 0; q < 2 * NP; q++) {
                next[q][0] += pcols;
                next[q][1] += pcols;
            }
        };
        auto advance = [&]() {
#pragma unroll
            for (int q = 0; q < NP; q++) {
                Ra[0][q] = Ra[1][q];
                Rb[0][q] = Rb[1][q];
            }
            load(1);
        };
        __syncwarp();
        load(0);
        load(1);
#pragma unroll
        for (int j = 0; j < UPW; j++) {
            if (j > 0) {
                if ((adv1 >> j) & 1) advance();
                if (A > 1 && ((adv2 >> j) & 1)) advance();
            }
            if (!((crosses >> j) & 1)) {
#pragma unroll
                for (int q = 0; q < NP; q++) acc[j][q] = f2_fma(tb[q], Ra[0][q], f2_fma(nb[q], Rb[0][q], acc[j][q]));
            } else {
                const f32x2 t = *reinterpret_cast<const f32x2*>(&s_ta[warp][j]);
                const float ts = s_ta[warp][j].x;
                const bool dn = (down >> j) & 1;
#pragma unroll
                for (int q = 0; q < NP; q++) {
                    // shares of (first row, j0), (first, j1), (second, j0), (second, j1)
                    const f32x2 w0 = f2_pack(fminf(ts, tbs[2 * q]), fminf(ts, tbs[2 * q + 1]));
                    const f32x2 w1 = f2_fma(minus, w0, t), w2 = f2_fma(minus, w0, tb[q]);
                    const f32x2 w3 = f2_fma(minus, f2_add(t, w2), one);
                    // a ray moving towards smaller x meets the higher row first
                    f32x2 s = acc[j][q];
                    if (dn) {
                        s = f2_fma(w0, Ra[1][q], f2_fma(w1, Rb[1][q], s));
                        s = f2_fma(w2, Ra[0][q], f2_fma(w3, Rb[0][q], s));
                    } else {
                        s = f2_fma(w0, Ra[0][q], f2_fma(w1, Rb[0][q], s));
                        s = f2_fma(w2, Ra[1][q], f2_fma(w3, Rb[1][q], s));
                    }
                    acc[j][q] = s;
                }
            }
        }
        pu += du;
#pragma unroll
        for (int q = 0; q < 2 * NP; q++) pv[q] += dv[q];
    }
    cp_async_wait<0>();
    // lengths per slab
    const double dx = cd.d[0], dy = cd.d[1], dz = cd.d[2];
#pragma unroll
    for (int q = 0; q < 2 * NP; q++) {
        const int iv = v0 + lane + 32 * q;
        const double rv = fma((double)iv, V.rv1, V.rv0) * dy, yz = fma(rv, rv, dz * dz);
#pragma unroll
        for (int j = 0; j < UPW; j++) {
            const int iu = uw + j;
            if (iu < cd.nu && iv < cd.nv) {
                const double rx = fma((double)iu, V.ru1, V.ru0) * dx;
                const float2 a = f2_unpack(acc[j][q / 2]);
                prj[bt * cd.prj_b + (((long long)iu * cd.nview + view) * cd.nv + iv) * cd.nc + c] =
                    (q & 1 ? a.y : a.x) * (float)sqrt(fma(rx, rx, yz));
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Backprojection.
// ---------------------------------------------------------------------------
// Projections of one (b, c) times the rays' lengths per slab, in rows of v:
// wp[view][u][pitch] (pitch = nv rounded up to 4, the padding zero); *bad set where
// one is not finite.  Block 256 along v; blockIdx = (v, u, view).
__global__ void __launch_bounds__(256) cone_tile_weight_kernel(float* __restrict__ wp, int* __restrict__ bad,
                                                               const float* __restrict__ prj,
                                                               const TileView* __restrict__ views, ConeDims cd,
                                                               int pitch, int bt, int c) {
    const int view = blockIdx.z, iu = blockIdx.y, iv = blockIdx.x * 256 + threadIdx.x;
    if (iv >= pitch) return;
    float val = 0.f;
    if (iv < cd.nv) {
        const TileView& V = views[view];
        const float ru = (float)fma((double)iu, V.ru1, V.ru0), rv = (float)fma((double)iv, V.rv1, V.rv0);
        const float seg =
            sqrtf(fmaf(ru * ru, cd.d[0] * cd.d[0], fmaf(rv * rv, cd.d[1] * cd.d[1], cd.d[2] * cd.d[2])));
        val = prj[bt * cd.prj_b + (((long long)iu * cd.nview + view) * cd.nv + iv) * cd.nc + c] * seg;
    }
    wp[((long long)view * cd.nu + iu) * pitch + iv] = val;
    if (!isfinite(val)) atomicOr(bad, 1);
}

constexpr int kBpXpw = 8, kBpTz = 4;                  // columns of voxels per warp, planes per block
constexpr int kBpTx = 4 * kBpXpw, kBpTy = 64;

// KV: rows iv that can meet one voxel (the host's bound).
template <int KV>
__global__ void __launch_bounds__(128, 3) cone_bp_tile_kernel(float* __restrict__ img, const float* __restrict__ wp,
                                                               const int* __restrict__ bad,
                                                               const TileView* __restrict__ views, ConeDims cd,
                                                               int pitch, int patch, int smem_bytes, int bt, int c,
                                                               int accumulate) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float4 s_ray[4][32];   // per warp: crossing time, patch row offset, voxel | flags
    __shared__ int4 s_win[4];         // per slot: first u, first v (a multiple of 4), columns (a multiple of 4), cut
    if (*bad) return;   // cone_bp_tile_direct_kernel's
    const int S = min(4, smem_bytes / (4 * patch));   // >= 2
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nx = cd.n[0], ny = cd.n[1], nz = cd.n[2];
    const int z0 = blockIdx.x * kBpTz, x0 = blockIdx.y * kBpTx, y0 = blockIdx.z * kBpTy;   // z fastest
    const int xw = x0 + warp * kBpXpw;
    auto issue = [&](int view, int slot) {
        // rays that meet the tile between its lowest and highest z face; ray i
        // meets a face at A + i G, A and G linear in z, so the outermost faces
        // bound the rest
        const TileView& V = views[view];
        float ulo = 1e30f, uhi = -1e30f, vlo = 1e30f, vhi = -1e30f;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const double M = (k ? z0 + kBpTz : z0) - V.sm;
            const float iu = __fdividef(1.f, (float)(M * V.ru1)), iv = __fdividef(1.f, (float)(M * V.rv1));
            const float au = (float)(x0 - fma(M, V.ru0, V.su)), av = (float)(y0 - fma(M, V.rv0, V.sv));
            ulo = fminf(ulo, au * iu);
            uhi = fmaxf(uhi, (au + kBpTx) * iu);
            vlo = fminf(vlo, av * iv);
            vhi = fmaxf(vhi, (av + kBpTy) * iv);
        }
        // the detector's own part of them
        const int ub = max((int)floorf(ulo - 0.01f), 0), vb = max((int)floorf(vlo - 0.01f), 0) & ~3;
        const int cols = (max(min((int)ceilf(vhi + 0.01f), cd.nv - 1) - vb, 0) + KV + 4) & ~3;
        int rows = min((int)ceilf(uhi + 0.01f), cd.nu - 1) - ub + 1;
        // (the host's patch holds every window, see cone_tile_views; were it ever smaller,
        // the tile would come out NaN)
        const bool cut = rows * cols > patch;
        if (cut) rows = patch / cols;
        if (threadIdx.x == 0) s_win[slot] = make_int4(ub, vb, cols, cut);
        const int j = vb + 4 * lane;
        const float* row = wp + ((long long)view * cd.nu + ub + warp) * pitch + j;
        const uint32_t dst = smem_u32(smem + slot * patch) + (warp * cols + 4 * lane) * 4;
        for (int q = 0; q < cols; q += 128) {
            if (4 * lane + q >= cols) break;
            const bool jin = j + q >= 0 && j + q < pitch;
            const float* s = row + q;
            uint32_t t = dst + 4 * q;
#pragma unroll 4
            for (int r = warp; r < rows; r += 4) {
                const bool in = jin && (unsigned)(ub + r) < (unsigned)cd.nu;
                cp_async16(t, in ? s : wp, in);
                s += 4 * pitch;
                t += 16 * cols;
            }
        }
    };
    f32x2 acc[kBpTz][kBpXpw];
#pragma unroll
    for (int z = 0; z < kBpTz; z++)
#pragma unroll
        for (int k = 0; k < kBpXpw; k++) acc[z][k] = 0ull;
    for (int s = 0; s < S - 1; s++) {
        if (s < cd.nview) issue(s, s);
        cp_async_commit();
    }
    int slot = 0, fill = S - 1;
    for (int view = 0; view < cd.nview; view++) {
        if (S == 2) cp_async_wait<0>();
        else if (S == 3) cp_async_wait<1>();
        else cp_async_wait<2>();
        __syncthreads();   // this view's patch is in; every warp has left the slot filled next
        if (view + S - 1 < cd.nview) issue(view + S - 1, fill);
        cp_async_commit();
        const TileView& V = views[view];
        const int4 win = s_win[slot];
        const int ub = win.x, vb = win.y, cols = win.z;
        if (win.w) {
            const float nan = __int_as_float(0x7fffffff);
#pragma unroll
            for (int z = 0; z < kBpTz; z++)
#pragma unroll
                for (int k = 0; k < kBpXpw; k++) acc[z][k] = f2_pack(nan, nan);
        }
        const float* pbase = smem + slot * patch;
#pragma unroll
        for (int z = 0; z < kBpTz; z++) {
            const double M = z0 + z - V.sm;
            // columns: lane k takes ray ia + k, ia the first that can meet the
            // warp's voxels
            const double gu0 = M * V.ru1, gu1 = gu0 + V.ru1;
            const double au0 = fma(M, V.ru0, V.su) - xw, au1 = au0 + V.ru0;   // ray 0 at the slab's two faces
            const float q0 = (float)-au0 * __fdividef(1.f, (float)gu0), q1 = (float)-au1 * __fdividef(1.f, (float)gu1);
            const int ia = (int)ceilf(fminf(q0, q1) - 1e-2f), iu = ia + lane;
            const long long p0 = to_fixed(fma((double)iu, gu0, au0)), p1 = to_fixed(fma((double)iu, gu1, au1));
            const int c0 = (int)(p0 >> 32), c1 = (int)(p1 >> 32), low = min(c0, c1);
            const float r = fabsf((float)(p1 - p0)) * 2.3283064365386963e-10f;
            const float ta = cross_time(p0, p1 - p0, __fdividef(1.f, fmaxf(r, 1e-30f)));
            const bool valid = (unsigned)iu < (unsigned)cd.nu && max(c0, c1) >= 0 && low < kBpXpw;
            const unsigned live = __ballot_sync(0xffffffffu, valid);
            __syncwarp();   // the previous plane's rays have been read
            s_ray[warp][lane] = make_float4(ta, __int_as_float((iu - ub) * cols),
                                            __int_as_float((low + 8) | (c0 != c1 ? 256 : 0) | (c1 < c0 ? 512 : 0)), 0.f);
            // rows: the first of the rays that can meet this lane's voxels and
            // the part of the slab each spends inside
            const double gv0 = M * V.rv1, gv1 = gv0 + V.rv1;
            const double av0 = fma(M, V.rv0, V.sv) - y0, av1 = av0 + V.rv0;
            const float ig0 = __fdividef(1.f, (float)gv0), ig1 = __fdividef(1.f, (float)gv1);
            const double bv0 = fma((double)vb, gv0, av0), bv1 = fma((double)vb, gv1, av1);   // ray vb at the two faces
            const float fb0 = (float)bv0, fb1 = (float)bv1;
            // 64-bit fixed point with 40 fractional bits; offsets from a voxel are
            // rounded to 26 and held to +-8 voxels (farther rays miss it either way)
            constexpr int kWide = 40, kBits = 26;
            constexpr float kUnit = 1.0f / (1 << kBits);
            auto wide = [](double v) { return llrint(v * (double)(1ll << kWide)); };
            const long long fx0 = wide(bv0), fx1 = wide(bv1), fg0 = wide(gv0), fg1 = wide(gv1);
            auto near = [](long long v) {
                constexpr long long kFar = 8ll << kWide, kHalf = 1ll << (kWide - kBits - 1);
                return (int)((max(min(v, kFar), -kFar) + kHalf) >> (kWide - kBits));
            };
            const int g0 = near(fg0), g1 = near(fg1), level = V.vt - vb;
            const float* col[2];
            f32x2 len[KV];
            float lo[2][KV], hi[2][KV];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int pv = lane + 32 * h;
                const float e0 = ((float)pv - fb0) * ig0, e1 = ((float)pv - fb1) * ig1;
                const int jl = min(max((int)ceilf(fminf(e0, e1) - 1e-3f), 0), cols - KV);
                col[h] = pbase + jl;
                const long long off = (long long)pv << kWide;
                // stepped from the level ray where the lane has it: in a voxel face it
                // must come out exactly there (then it belongs to the voxel above, as in
                // the forward projection)
                const int jb = min(max(level, jl), jl + KV - 1);
                const int x0i = near(fx0 + jb * fg0 - off) - (jb - jl) * g0, x1i = near(fx1 + jb * fg1 - off) - (jb - jl) * g1;
#pragma unroll
                for (int k = 0; k < KV; k++) {
                    // offsets at the two faces, the slope, and the times at 0 and 1
                    const float xa = (float)(x0i + k * g0) * kUnit;
                    const float rr = (float)((x1i - x0i) + k * (g1 - g0)) * kUnit;
                    const float ir = fabsf(rr) > 1e-30f ? __fdividef(1.f, rr) : 1e30f;
                    const float s0 = -xa * ir, s1 = (1.f - xa) * ir;
                    lo[h][k] = fmaxf(fminf(s0, s1), 0.f);
                    hi[h][k] = fmaxf(fminf(fmaxf(s0, s1), 1.f), lo[h][k]);
                }
            }
#pragma unroll
            for (int k = 0; k < KV; k++) len[k] = f2_pack(hi[0][k] - lo[0][k], hi[1][k] - lo[1][k]);
            __syncwarp();
            // walk the columns
            const f32x2 minus = f2_pack(-1.f, -1.f);
            int k = live ? __ffs(live) - 1 : 0;
            const int kend = live ? 32 - __clz(live) : 0;
            f32x2 carry = 0ull;
            auto ray = [&](f32x2& here, int flags, float t, int o) {
                f32x2 P[KV];
                f32x2 full;
#pragma unroll
                for (int i = 0; i < KV; i++) {
                    P[i] = f2_pack(col[0][o + i], col[1][o + i]);
                    full = i ? f2_fma(len[i], P[i], full) : f2_mul(len[i], P[i]);
                }
                if (!(flags & 256)) {
                    here = f2_add(here, full);
                } else {
                    f32x2 part = 0ull;
#pragma unroll
                    for (int i = 0; i < KV; i++) {
                        const f32x2 l = f2_pack(fmaxf(fminf(hi[0][i], t) - lo[0][i], 0.f),
                                                fmaxf(fminf(hi[1][i], t) - lo[1][i], 0.f));
                        part = f2_fma(l, P[i], part);
                    }
                    const f32x2 rest = f2_fma(minus, part, full);
                    // towards larger x the lower voxel comes first
                    if (flags & 512) {
                        here = f2_add(here, rest);
                        carry = f2_add(carry, part);
                    } else {
                        here = f2_add(here, part);
                        carry = f2_add(carry, rest);
                    }
                }
            };
            float4 e = s_ray[warp][min(k, 31)];
            {   // columns that come from the voxel before the warp's first
                f32x2 gone = 0ull;
                while (k < kend && (__float_as_int(e.z) & 255) < 8) {
                    ray(gone, __float_as_int(e.z), e.x, __float_as_int(e.y));
                    k++;
                    e = s_ray[warp][min(k, 31)];
                }
            }
#pragma unroll
            for (int j = 0; j < kBpXpw; j++) {
                f32x2 s = carry;
                carry = 0ull;
                while (k < kend && (__float_as_int(e.z) & 255) == 8 + j) {
                    ray(s, __float_as_int(e.z), e.x, __float_as_int(e.y));
                    k++;
                    e = s_ray[warp][min(k, 31)];
                }
                acc[z][j] = f2_add(acc[z][j], s);
            }
        }
        slot = slot + 1 == S ? 0 : slot + 1;
        fill = fill + 1 == S ? 0 : fill + 1;
    }
    cp_async_wait<0>();
#pragma unroll
    for (int j = 0; j < kBpXpw; j++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int ix = xw + j, iy = y0 + lane + 32 * h;
            if (ix < nx && iy < ny) {
                float v[kBpTz];
#pragma unroll
                for (int z = 0; z < kBpTz; z++) {
                    const float2 a = f2_unpack(acc[z][j]);
                    v[z] = h ? a.y : a.x;
                }
                float* out = img + bt * cd.img_b + (long long)ix * cd.st[0] + (long long)iy * cd.st[1] +
                             (long long)z0 * cd.nc + c;
                if (cd.nc == 1 && !accumulate && z0 + kBpTz <= nz && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
                    *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int z = 0; z < kBpTz; z++)
                        if (z0 + z < nz) {
                            float* o = out + (long long)z * cd.nc;
                            *o = accumulate ? *o + v[z] : v[z];
                        }
                }
            }
        }
}

// The slice whose projections hold a value that is not finite, a voxel per thread.
// The tiles add rows of rays that miss a voxel with a length of 0, which would make NaN
// of it; here only the rays that meet a voxel count, each by its length.
__device__ __forceinline__ bool direct_interval(double a0, double a1, double& t0, double& t1) {
    // positions at the two faces, as the forward projection rounds them
    a0 = rint(a0 * 4294967296.0) / 4294967296.0;
    a1 = rint(a1 * 4294967296.0) / 4294967296.0;
    t0 = 0.0;
    t1 = 1.0;
    if (a0 == a1) return a0 >= 0.0 && a0 < 1.0;
    const double p = -a0 / (a1 - a0), q = (1.0 - a0) / (a1 - a0);
    t0 = fmax(t0, fmin(p, q));
    t1 = fmin(t1, fmax(p, q));
    return t1 > t0;
}

__global__ void __launch_bounds__(256) cone_bp_tile_direct_kernel(float* __restrict__ img, const float* __restrict__ wp,
                                                                  const int* __restrict__ bad,
                                                                  const TileView* __restrict__ views, ConeDims cd,
                                                                  int pitch, int bt, int c, int accumulate) {
    if (*bad == 0) return;
    const long long n = (long long)cd.n[0] * cd.n[1] * cd.n[2];
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
        const int z = (int)(i % cd.n[2]), y = (int)(i / cd.n[2] % cd.n[1]), x = (int)(i / cd.n[2] / cd.n[1]);
        float acc = 0.f;
        for (int view = 0; view < cd.nview; view++) {
            const TileView& V = views[view];
            // ray i lies at a + i g on the voxel's two faces (relative to it)
            const double M0 = z - V.sm, M1 = M0 + 1.0;
            const double au0 = fma(M0, V.ru0, V.su) - x, au1 = fma(M1, V.ru0, V.su) - x, gu0 = M0 * V.ru1, gu1 = M1 * V.ru1;
            const double av0 = fma(M0, V.rv0, V.sv) - y, av1 = fma(M1, V.rv0, V.sv) - y, gv0 = M0 * V.rv1, gv1 = M1 * V.rv1;
            const int i0 = max(0, (int)floor(fmin(-au0 / gu0, -au1 / gu1)) - 1);
            const int i1 = min(cd.nu - 1, (int)ceil(fmax((1.0 - au0) / gu0, (1.0 - au1) / gu1)) + 1);
            const int j0 = max(0, (int)floor(fmin(-av0 / gv0, -av1 / gv1)) - 1);
            const int j1 = min(cd.nv - 1, (int)ceil(fmax((1.0 - av0) / gv0, (1.0 - av1) / gv1)) + 1);
            for (int iu = i0; iu <= i1; iu++) {
                double t0, t1;
                if (!direct_interval(fma((double)iu, gu0, au0), fma((double)iu, gu1, au1), t0, t1)) continue;
                const float* row = wp + ((long long)view * cd.nu + iu) * pitch;
                for (int iv = j0; iv <= j1; iv++) {
                    double s0, s1;
                    if (!direct_interval(fma((double)iv, gv0, av0), fma((double)iv, gv1, av1), s0, s1)) continue;
                    const double len = fmin(t1, s1) - fmax(t0, s0);
                    if (len > 1e-9) acc = fmaf((float)len, row[iv], acc);
                }
            }
        }
        float* o = img + bt * cd.img_b + (long long)x * cd.st[0] + (long long)y * cd.st[1] + (long long)z * cd.nc + c;
        *o = accumulate ? *o + acc : acc;
    }
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
// The limits: z the main axis of every view, u along +x and v along +y; the
// source and the detector on opposite sides of all slabs; slopes of at most one
// voxel per slab; rays spaced 0.3 to 1.9 voxels (FP tiles, the 32 rays of a
// warp's voxels); at most 4 rows of rays over a voxel; patches that fit in
// shared memory twice.
bool cone_tile_views(const std::vector<ConeView>& views, const ConeDims& cd, std::vector<TileView>& out,
                     TilePlan& tp) {
    out.clear();
    const double nz = cd.n[2];
    double gu_lo = 1e300, gu_hi = 0, gv_lo = 1e300, gv_hi = 0, ru_hi = 0, rv_hi = 0, far = 0;
    if (cd.nview > 65535 || cd.nu > 65535) return false;
    for (const ConeView& v : views) {
        if (v.affine != 1 || v.m != 2 || v.a != 0 || v.b != 1) return false;
        TileView q;
        q.su = v.S[0];
        q.sv = v.S[1];
        q.sm = v.S[2];
        q.ru0 = v.rho[0];
        q.ru1 = v.rho[1];
        q.rv0 = v.rho[3];
        q.rv1 = v.rho[5];
        q.vt = (int)std::min(std::max(std::rint(-q.rv0 / q.rv1), -1e9), 1e9);
        const double e = q.sm + v.Dm0;
        if (!((q.sm < -0.5 && e >= nz) || (q.sm > nz + 0.5 && e <= 0.0))) return false;
        double glo[2] = {1e300, 1e300}, ghi[2] = {0, 0};
        for (double pm : {0.0, nz}) {   // spacing at the outermost faces
            const double g[2] = {(pm - q.sm) * q.ru1, (pm - q.sm) * q.rv1};
            for (int k = 0; k < 2; k++) {
                glo[k] = std::min(glo[k], g[k]);
                ghi[k] = std::max(ghi[k], g[k]);
            }
            for (double i : {0.0, (double)cd.nu + 256}) far = std::max(far, std::fabs(q.su + (pm - q.sm) * (q.ru0 + i * q.ru1)));
            for (double i : {0.0, (double)cd.nv + 256}) far = std::max(far, std::fabs(q.sv + (pm - q.sm) * (q.rv0 + i * q.rv1)));
        }
        if (!(glo[0] > 0.0 && glo[1] > 0.0)) return false;
        for (double i : {0.0, cd.nu - 1.0}) ru_hi = std::max(ru_hi, std::fabs(q.ru0 + i * q.ru1));
        for (double i : {0.0, cd.nv - 1.0}) rv_hi = std::max(rv_hi, std::fabs(q.rv0 + i * q.rv1));
        // one slab more on both sides than there is: the last block's planes
        q.gu_max = (float)ghi[0];
        q.gv_max = (float)ghi[1];
        gu_lo = std::min(gu_lo, glo[0]);
        gu_hi = std::max(gu_hi, ghi[0]);
        gv_lo = std::min(gv_lo, glo[1]);
        gv_hi = std::max(gv_hi, ghi[1]);
        out.push_back(q);
    }
    if (!(ru_hi <= 1.0 && rv_hi <= 1.0 && gu_lo >= 0.3 && gv_lo >= 0.3 && gu_hi <= kTileWide && gv_hi <= kTileWide &&
          far < 1e4))
        return false;
    // the last block of planes reaches up to kBpTz - 1 slabs beyond the volume
    for (const TileView& q : out)
        if (!(std::fabs(nz + kBpTz - q.sm) > 0.5 && (nz + kBpTz - q.sm) * (nz - q.sm) > 0)) return false;
    double lo_u = gu_lo, lo_v = gv_lo;
    for (const TileView& q : out) {
        lo_u = std::min(lo_u, (nz + kBpTz - q.sm) * q.ru1);
        lo_v = std::min(lo_v, (nz + kBpTz - q.sm) * q.rv1);
    }
    if (!(lo_u >= 0.28 && lo_v >= 0.28)) return false;
    if ((kBpXpw + 1.0) / lo_u + 2.0 > 32.0) return false;   // rays of a warp's voxels
    tp.kv = (int)std::floor((1.0 + rv_hi + 2e-2) / lo_v) + 1;
    if (tp.kv > 4) return false;
    tp.kv = std::max(tp.kv, 3);
    const int kv = tp.kv;
    // Backprojection window of a tile.  Of the detector's rays those between the
    // lowest and the highest that meet it count; two of them that cross its faces at
    // m0 and m1, x0 and x1 apart, lie (x1 - x0 - r (m1 - m0)) / g1 apart, r <= ru_hi the
    // slope of one and g1 the spacing at m1: at most (kBpTx + kBpTz ru_hi) / lo_u.  The
    // kernel adds 0.02 for its FP32 arithmetic and rounds outwards, which is under 3.1
    // rows more (4 and a row here), along v to a multiple of 4 before and after, under
    // 9.1 + KV (10 + kv and 3 here).
    const double rows = (kBpTx + kBpTz * ru_hi) / lo_u + 4.0, cols = (kBpTy + kBpTz * rv_hi) / lo_v + kv + 10.0;
    tp.bp_patch = ((int)rows + 1) * (((int)cols + 4) & ~3);
    if (8LL * tp.bp_patch > kBpTileSmemWide) return false;
    tp.bp_smem = 8 * tp.bp_patch > kBpTileSmem ? kBpTileSmemWide : kBpTileSmem;
    tp.fp_narrow = gu_hi <= kTileNarrow && gv_hi <= kTileNarrow;
    tp.gu = gu_hi;
    tp.gv = gv_hi;
    return true;
}

static std::mutex g_tile_mu;
static std::vector<char> g_tile_done;
int cone_tile_attributes() {
    int dev = 0;
    RN_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_tile_mu);
    if ((int)g_tile_done.size() <= dev) g_tile_done.resize(dev + 1, 0);
    if (g_tile_done[dev]) return RN_OK;
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    RN_CUDA_TRY(cudaFuncSetAttribute(cone_fp_tile_kernel<1, 16, 2>, attr, kFpTileSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(cone_fp_tile_kernel<2, 8, 1>, attr, kFpTileSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(cone_bp_tile_kernel<3>, attr, kBpTileSmemWide));
    RN_CUDA_TRY(cudaFuncSetAttribute(cone_bp_tile_kernel<4>, attr, kBpTileSmemWide));
    g_tile_done[dev] = 1;
    return RN_OK;
}

size_t cone_tile_fp_bytes(const ConeDims& cd) {
    return sizeof(float) * (size_t)cd.n[2] * cd.n[0] * ((cd.n[1] + 3) & ~3);
}
static size_t tile_bp_floats(const ConeDims& cd) { return (size_t)cd.nview * cd.nu * ((cd.nv + 3) & ~3); }
size_t cone_tile_bp_bytes(const ConeDims& cd) { return sizeof(float) * (tile_bp_floats(cd) + 1); }   // and the flag

// Tiles of 64 x 128 rays for rays under a voxel apart where they fill the GPU.
bool cone_tile_big(const ConeDims& cd, const TilePlan& tp) {
    return tp.fp_narrow && (long long)((cd.nu + 63) / 64) * ((cd.nv + 127) / 128) * cd.nview >= 3 * 148;
}

int cone_tile_project(const TileView* d_views, const ConeDims& cd, const TilePlan& tp, float* d_vol, float* d_prj,
                      const float* d_img, cudaStream_t st) {
    const int pitch = (cd.n[1] + 3) & ~3;
    const bool big = cone_tile_big(cd, tp);
    for (int b = 0; b < cd.nb; b++)
        for (int c = 0; c < cd.nc; c++) {
            cone_planes_kernel<<<dim3((pitch + 31) / 32, (cd.n[2] + 31) / 32, std::min(cd.n[0], 64)), dim3(32, 8), 0,
                                 st>>>(d_vol, d_img, cd, pitch, b, c);
            if (big)
                cone_fp_tile_kernel<1, 16, 2><<<dim3((cd.nv + 127) / 128, (cd.nu + 63) / 64, cd.nview), 128,
                                                kFpTileSmem, st>>>(d_prj, d_vol, d_views, cd, pitch, b, c);
            else
                cone_fp_tile_kernel<2, 8, 1><<<dim3((cd.nv + 63) / 64, (cd.nu + 31) / 32, cd.nview), 128, kFpTileSmem,
                                               st>>>(d_prj, d_vol, d_views, cd, pitch, b, c);
        }
    RN_CUDA_TRY(cudaGetLastError());
    return RN_OK;
}

int cone_tile_backproject(const TileView* d_views, const ConeDims& cd, const TilePlan& tp, float* d_wp, float* d_img,
                          const float* d_prj, int accumulate, cudaStream_t st) {
    const int pitch = (cd.nv + 3) & ~3;
    int* d_bad = reinterpret_cast<int*>(d_wp + tile_bp_floats(cd));
    const dim3 grid((unsigned)((cd.n[2] + kBpTz - 1) / kBpTz), (unsigned)((cd.n[0] + kBpTx - 1) / kBpTx),
                    (unsigned)((cd.n[1] + kBpTy - 1) / kBpTy));
    for (int b = 0; b < cd.nb; b++)
        for (int c = 0; c < cd.nc; c++) {
            RN_CUDA_TRY(cudaMemsetAsync(d_bad, 0, sizeof(int), st));
            cone_tile_weight_kernel<<<dim3((pitch + 255) / 256, cd.nu, cd.nview), 256, 0, st>>>(d_wp, d_bad, d_prj, d_views,
                                                                                                cd, pitch, b, c);
            if (tp.kv <= 3)
                cone_bp_tile_kernel<3><<<grid, 128, tp.bp_smem, st>>>(d_img, d_wp, d_bad, d_views, cd, pitch, tp.bp_patch,
                                                                      tp.bp_smem, b, c, accumulate);
            else
                cone_bp_tile_kernel<4><<<grid, 128, tp.bp_smem, st>>>(d_img, d_wp, d_bad, d_views, cd, pitch, tp.bp_patch,
                                                                      tp.bp_smem, b, c, accumulate);
            cone_bp_tile_direct_kernel<<<148 * 8, 256, 0, st>>>(d_img, d_wp, d_bad, d_views, cd, pitch, b, c, accumulate);
        }
    RN_CUDA_TRY(cudaGetLastError());
    return RN_OK;
}

}  // namespace rn
