// Tomosynthesis distance-driven projector pair (flat detector with detU = x,
// detV = y, main axis z), restating DistanceDrivenTomo::ProjectionTomo /
// BackprojectionTomo (ReconNet4D/DistanceDriven3D.cu:37-663):
//   FP: per ray, for every z plane at integer z, the source-to-detector
//       rectangle [x1,x2] x [y1,y2] spanned by the cell's edge rays is
//       integrated over the piecewise-constant plane (the reference reads 4
//       bilinear corners of a 2D summed-area table), normalised by its area,
//       and the sum is scaled by dz / |dz_src-det| * |src - det|;
//   BP: the sinogram is pre-weighted by the same length factor, and every
//       voxel integrates the detector rectangle spanned by its projected faces.
// Both integrals are separable: on a plane the rectangle is an x interval that
// depends on the cell's u only times a y interval that depends on its v only.
// The tile kernels (tomo_fp_tile_kernel, tomo_bp_tile_kernel) use that: the
// overlaps with the few voxels (cells) under a footprint are worked out once
// per u and once per v of a tile, in FP64, and the values are read from a
// patch staged in shared memory.  Geometries outside their limits (footprints
// wider than 1.9 voxels or 3 cells, the source between planes, a detector beyond
// the source) take the table kernels: the FP from FP64 row-prefix tables
// (rows_integral), the BP from the FP64 (u, v) summed-area table with the
// corners shared between neighbouring voxels.  The geometry arrays live on the
// device, so the choice is made there, by the same test in every kernel of the
// launch sequence.  Each (b, c) volume is processed by one launch sequence on
// the caller's stream.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <climits>
#include <mutex>
#include <vector>

#include "rn_device.cuh"
#include "rn_internal.h"

namespace rn {

struct TomoDims {
    int nb, nc, nx, ny, nz;
    float dx, dy, dz, cx, cy, cz;
    int nu, nview, nv;
    float du, dv, off_u, off_v;
};

// ---------------------------------------------------------------------------
// Separable footprints.
//
// In voxel units the left edge of detector column u meets the plane iz at
// x(u) = sx + (rx0 + u drx) (iz - sz), so on a plane every cell covers an
// interval of width drx (iz - sz); the same for v along y.  A voxel's faces
// fall on the detector at u(x) = A + r(z) (x - sp), r = (det - src) / (z - src).
// ---------------------------------------------------------------------------
struct TomoFpGeo {
    double sx, rx0, drx;   // x(u, iz) = sx + (rx0 + u drx) (iz - sz)
    double sy, ry0, dry;
    double sz;
};

__device__ __forceinline__ TomoFpGeo tomo_fp_geo(const TomoDims& d, const float* dc, const float* sp) {
    TomoFpGeo g;
    const double hx = d.nx / 2.0, hy = d.ny / 2.0, hz = d.nz / 2.0;
    g.sx = ((double)sp[0] - d.cx) / d.dx + hx;
    g.sy = ((double)sp[1] - d.cy) / d.dy + hy;
    g.sz = ((double)sp[2] - d.cz) / d.dz + hz;
    const double iz = 1.0 / (((double)dc[2] - d.cz) / d.dz + hz - g.sz);
    const double u0 = (-0.5 - d.off_u - (d.nu - 1) / 2.0) * d.du, v0 = (-0.5 - d.off_v - (d.nv - 1) / 2.0) * d.dv;
    g.rx0 = ((dc[0] + u0 - d.cx) / d.dx + hx - g.sx) * iz;
    g.ry0 = ((dc[1] + v0 - d.cy) / d.dy + hy - g.sy) * iz;
    g.drx = (double)d.du / d.dx * iz;
    g.dry = (double)d.dv / d.dy * iz;
    return g;
}
__device__ __forceinline__ double tomo_edge(double s, double r0, double dr, int e, double t) {
    return fma(fma((double)e, dr, r0), t, s);
}

// How many voxels a cell's footprint can touch per axis on any plane of this
// view: 2 (footprints at most kTomoNarrow wide), 3 (at most kTomoWide), or 0
// where the tile kernel does not apply.  The limits, a little under 1 and 2
// voxels, are the widths for which two patches fit in a block's shared memory.
constexpr double kTomoNarrow = 0.95, kTomoWide = 1.9;
__device__ __forceinline__ int tomo_fp_class(const TomoDims& d, const float* dc, const float* sp) {
    const TomoFpGeo g = tomo_fp_geo(d, dc, sp);
    const double t0 = -g.sz, t1 = d.nz - 1 - g.sz;
    if (!(t0 * t1 > 0)) return 0;   // the source between the planes (or not a number)
    const double lo = fmin(fmin(g.drx * t0, g.drx * t1), fmin(g.dry * t0, g.dry * t1));
    const double hi = fmax(fmax(g.drx * t0, g.drx * t1), fmax(g.dry * t0, g.dry * t1));
    if (!(lo > 1e-3 && hi <= kTomoWide)) return 0;
    double far = 0.0;
    for (int k = 0; k < 2; k++) {
        const double t = k ? t1 : t0;
        far = fmax(far, fmax(fabs(tomo_edge(g.sx, g.rx0, g.drx, 0, t)), fabs(tomo_edge(g.sx, g.rx0, g.drx, d.nu, t))));
        far = fmax(far, fmax(fabs(tomo_edge(g.sy, g.ry0, g.dry, 0, t)), fabs(tomo_edge(g.sy, g.ry0, g.dry, d.nv, t))));
    }
    if (!(far < 1e6)) return 0;
    return hi <= kTomoNarrow ? 2 : 3;
}

// Which kernels a call needs, decided once per call by a kernel of its own (in the
// others the test costs 2 to 4 us each, and registers) and kept in the scratch's first double.  That entry of the tables
// is zero, so the word keeps its meaning while they are built:
//   forward: 4 and / or 8 where every view has class 2 or 3 (the tile kernels), 0 where
//     every view has class 0 (the tables), -0.0 where only some have (both);
//   back: the call's class and patch, or 0 (the tables).
constexpr unsigned long long kTomoMixed = 1ull << 63;
__device__ __forceinline__ unsigned long long tomo_word(const double* sat) {
    return *reinterpret_cast<const volatile unsigned long long*>(sat);
}

__global__ void __launch_bounds__(128) tomo_fp_decide(double* sat, const float* __restrict__ detCenter,
                                                      const float* __restrict__ src, TomoDims d) {
    int found = 0;
    for (int v = threadIdx.x; v < d.nview; v += 128) found |= 1 << tomo_fp_class(d, detCenter + 3 * v, src + 3 * v);
    const bool c0 = __syncthreads_or(found & 1), c2 = __syncthreads_or(found & 4), c3 = __syncthreads_or(found & 8);
    if (threadIdx.x == 0)
        *reinterpret_cast<unsigned long long*>(sat) = c0 ? (c2 || c3 ? kTomoMixed : 0ull) : (c2 ? 4ull : 0ull) | (c3 ? 8ull : 0ull);
}

// Overlaps of an interval that starts a fraction f into a unit cell and is
// `width` wide (at most K - 1) with the K cells from there on, as shares of
// the width.
template <int K>
__device__ __forceinline__ void taps_at(float f, float width, float (&w)[K]) {
    const float iw = __fdividef(1.0f, width);
    float rest = width, o = fminf(1.0f - f, rest);
    w[0] = o * iw;
#pragma unroll
    for (int k = 1; k < K - 1; k++) {
        rest -= o;
        o = fminf(1.0f, rest);
        w[k] = o * iw;
    }
    w[K - 1] = (rest - o) * iw;
}

// Positions as 64-bit fixed point (32 fractional bits).
__device__ __forceinline__ long long tomo_fixed(double v) { return llrint(v * 4294967296.0); }
__device__ __forceinline__ float tomo_frac(long long p) { return __uint2float_rn((unsigned)p) * 2.3283064365386963e-10f; }

// Values of 2 NP lanes' columns walked together: NP pairs of rows R[k], k < K,
// the lane's v-weighted sums of K consecutive patch rows; `next` points at the
// patch row loaded next, per lane.
template <int K, int NP>
struct RowWalk {
    f32x2 R[K][NP], t[K][NP];
    const float* next[2 * NP];
    int stride;
    __device__ __forceinline__ void load(int slot) {
#pragma unroll
        for (int q = 0; q < NP; q++) {
            const float *a = next[2 * q], *b = next[2 * q + 1];
            f32x2 s = f2_mul(t[0][q], f2_pack(a[0], b[0]));
#pragma unroll
            for (int k = 1; k < K; k++) s = f2_fma(t[k][q], f2_pack(a[k], b[k]), s);
            R[slot][q] = s;
            next[2 * q] += stride;
            next[2 * q + 1] += stride;
        }
    }
    __device__ __forceinline__ void start() {
#pragma unroll
        for (int k = 0; k < K; k++) load(k);
    }
    __device__ __forceinline__ void advance() {
#pragma unroll
        for (int k = 0; k < K - 1; k++)
#pragma unroll
            for (int q = 0; q < NP; q++) R[k][q] = R[k + 1][q];
        load(K - 1);
    }
};

// The taps along the walked axis, as the walk reads them: every share twice
// (both halves of a pair).
template <int K>
struct WalkTaps {
    float4 a;                          // w0 w0 w1 w1
    float4 b[1];                       // w2 w2 w3 w3
};
template <>
struct WalkTaps<2> {
    float4 a;
};
__device__ __forceinline__ void store_taps(WalkTaps<2>& d, const float (&w)[2]) {
    d.a = make_float4(w[0], w[0], w[1], w[1]);
}
template <int K>
__device__ __forceinline__ void store_taps(WalkTaps<K>& d, const float (&w)[K]) {
    const float w3 = K > 3 ? w[K - 1] : 0.f;
    d.a = make_float4(w[0], w[0], w[1], w[1]);
    d.b[0] = make_float4(w[2], w[2], w3, w3);
}
template <int NP>
__device__ __forceinline__ void add_taps(const WalkTaps<2>& w, const RowWalk<2, NP>& r, f32x2 (&acc)[NP]) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(&w.a);
#pragma unroll
    for (int q = 0; q < NP; q++) acc[q] = f2_fma(a.y, r.R[1][q], f2_fma(a.x, r.R[0][q], acc[q]));
}
template <int K, int NP>
__device__ __forceinline__ void add_taps(const WalkTaps<K>& w, const RowWalk<K, NP>& r, f32x2 (&acc)[NP]) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(&w.a), b = *reinterpret_cast<const ulonglong2*>(&w.b[0]);
#pragma unroll
    for (int q = 0; q < NP; q++) {
        f32x2 s = f2_fma(a.y, r.R[1][q], f2_fma(a.x, r.R[0][q], acc[q]));
        s = f2_fma(b.x, r.R[2][q], s);
        acc[q] = K > 3 ? f2_fma(b.y, r.R[K - 1][q], s) : s;
    }
}

// Length weight of detector cell (u, v) of a view (PreweightBPCartKernelXY,
// DistanceDriven3D.cu:409-431).
__device__ __forceinline__ double tomo_len_weight(const float* dc, const float* sp, float u, float v, float dz) {
    const double ddx = (double)sp[0] - (dc[0] + u), ddy = (double)sp[1] - (dc[1] + v), ddz = (double)sp[2] - dc[2];
    return (double)dz / fabs(ddz) * sqrt(ddx * ddx + ddy * ddy + ddz * ddz);
}

// Plane-major copy of one (b, c) volume for the tile kernel: vol[z][x][pitch],
// y fastest, pitch = ny rounded up to 4, the padding zero.  32 x 32 (y, z)
// tiles through shared memory.  Block (32, 8): blockIdx = (y tile, z tile, x).
__global__ void __launch_bounds__(256) tomo_planes_kernel(float* __restrict__ vol, const float* __restrict__ img,
                                                          const double* sat, TomoDims d, int pitch, int b, int c) {
    if (tomo_word(sat) == 0) return;   // no view for the tile kernels
    __shared__ float tile[32][33];
    const int y0 = blockIdx.x * 32, z0 = blockIdx.y * 32;
    const int lane = threadIdx.x, w = threadIdx.y;
    for (int x = blockIdx.z; x < d.nx; x += gridDim.z) {
        const float* base = img + ((long long)b * d.nx + x) * d.ny * d.nz * d.nc + c;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int y = y0 + w + 8 * k, z = z0 + lane;
            tile[w + 8 * k][lane] = (y < d.ny && z < d.nz) ? base[((long long)y * d.nz + z) * d.nc] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int z = z0 + w + 8 * k, y = y0 + lane;
            if (z < d.nz && y < pitch) vol[((long long)z * d.nx + x) * pitch + y] = tile[lane][w + 8 * k];
        }
        __syncthreads();
    }
}

// Forward projection of the views of class K (and, with `all`, of lower
// classes).  A block of 4 warps owns a tile of 4 UPW x 64 NP cells of one
// view; a warp UPW columns u by all rows v, lane l the rows l, l + 32, ...
// Plane after plane the patch of voxels under the tile arrives in shared
// memory (cp.async, 2 to 4 planes in flight).  Positions step from plane to
// plane in 64-bit fixed point.  A lane keeps the taps of its rows v in
// registers, lane j works out the taps of column u0 + j into shared memory.
// The warp then walks its columns: R[k] holds the v-weighted sums of the K
// voxel rows under the current column, which move on by at most K - 1 rows per
// column (the same for the whole warp: ballots), so a voxel row is read once
// per warp (K reads per lane and v) and a column costs K packed FMAs per two v.
// Bound by instruction issue (14 warp instructions per 32 ray-planes, 57% issue
// active).  512x512x128 voxels, 736x736 cells, 25 views: 1.20 ms (1.27 while
// warps beyond the detector's last column worked too), where the prefix-table
// kernel takes 6.66 ms (98 instructions: FP64 prefixes and positions worked out
// per ray and plane).
constexpr int kTomoTileSmem = 70 * 1024;   // with the static tables, three blocks per SM

template <int K, int UPW, int NP>
__global__ void __launch_bounds__(128, 3)
    tomo_fp_tile_kernel(float* __restrict__ prj, const float* __restrict__ vol, const double* sat,
                        const float* __restrict__ detCenter, const float* __restrict__ src, TomoDims d, int pitch, int b,
                        int c, int all) {
    constexpr int TU = 4 * UPW, TV = 64 * NP;
    constexpr double kWidest = K == 2 ? kTomoNarrow : kTomoWide;
    constexpr int kMaxRows = (int)(TU * kWidest) + K + 2, kMaxPitch = ((int)(TV * kWidest) + K + 2 + 6) & ~3;
    static_assert(2 * kMaxRows * kMaxPitch * 4 <= kTomoTileSmem, "two patches fit");
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(16) WalkTaps<K> s_ut[4][UPW];   // per warp; rewritten after the next barrier
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int u0 = blockIdx.y * TU, v0 = blockIdx.x * TV;
    const int uw = u0 + warp * UPW;
    const unsigned long long word = tomo_word(sat);
    if (word == 0 || (!all && word != kTomoMixed && !((word >> K) & 1))) return;
    for (int view = blockIdx.z; view < d.nview; view += gridDim.z) {
        const float* dc = detCenter + 3 * view;
        const float* sp = src + 3 * view;
        const int cls = tomo_fp_class(d, dc, sp);
        if (cls != K && !(all && cls && cls < K)) continue;   // block-uniform
        const TomoFpGeo g = tomo_fp_geo(d, dc, sp);
        // footprint widths on plane iz: wx + iz dwx, wy + iz dwy; patch
        // extents at the widest plane, and how many patches fit
        const double wmx = fmax(-g.sz * g.drx, (d.nz - 1 - g.sz) * g.drx);
        const double wmy = fmax(-g.sz * g.dry, (d.nz - 1 - g.sz) * g.dry);
        const float wx = (float)(-g.sz * g.drx), dwx = (float)g.drx, wy = (float)(-g.sz * g.dry), dwy = (float)g.dry;
        const int prows = min(kMaxRows, (int)(TU * wmx) + K + 2), pcols = min(kMaxPitch, ((int)(TV * wmy) + K + 2 + 6) & ~3);
        const int patch = prows * pcols;
        const int S = min(4, kTomoTileSmem / (4 * patch));   // >= 2
        // fixed-point positions at the current plane and their steps: lower
        // edges of the tile's first u and v, of this lane's column (for the
        // taps along u) and of its rows v
        long long pu0 = tomo_fixed(tomo_edge(g.sx, g.rx0, g.drx, u0, -g.sz)), du0 = tomo_fixed(fma((double)u0, g.drx, g.rx0));
        long long pv0 = tomo_fixed(tomo_edge(g.sy, g.ry0, g.dry, v0, -g.sz)), dv0 = tomo_fixed(fma((double)v0, g.dry, g.ry0));
        long long pu = tomo_fixed(tomo_edge(g.sx, g.rx0, g.drx, uw + lane % UPW, -g.sz));
        const long long du = tomo_fixed(fma((double)(uw + lane % UPW), g.drx, g.rx0));
        long long pv[2 * NP], dv[2 * NP];
#pragma unroll
        for (int q = 0; q < 2 * NP; q++) {
            pv[q] = tomo_fixed(tomo_edge(g.sy, g.ry0, g.dry, v0 + lane + 32 * q, -g.sz));
            dv[q] = tomo_fixed(fma((double)(v0 + lane + 32 * q), g.dry, g.ry0));
        }
        auto issue = [&](int iz, int slot) {
            const int ib = (int)((pu0 + iz * du0) >> 32), jb = (int)((pv0 + iz * dv0) >> 32) & ~3;
            const int j = jb + 4 * lane;
            const float* row = vol + ((long long)iz * d.nx + ib + warp) * pitch + j;
            const uint32_t dst = smem_u32(smem + slot * patch) + (warp * pcols + 4 * lane) * 4;
            for (int q = 0; q < pcols; q += 128) {
                if (4 * lane + q >= pcols) break;
                const bool jin = j + q >= 0 && j + q < pitch;
                const float* s = row + q;
                uint32_t t = dst + 4 * q;
#pragma unroll 4
                for (int r = warp; r < prows; r += 4) {
                    const bool in = jin && (unsigned)(ib + r) < (unsigned)d.nx;
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
            if (s < d.nz) issue(s, s);
            cp_async_commit();
        }
        int slot = 0, fill = S - 1;
        for (int iz = 0; iz < d.nz; iz++) {
            if (S == 2) cp_async_wait<0>();
            else if (S == 3) cp_async_wait<1>();
            else cp_async_wait<2>();
            __syncthreads();   // plane iz is in; every warp has left the slot filled next
            if (iz + S - 1 < d.nz) issue(iz + S - 1, fill);
            cp_async_commit();
            const int now = slot;
            slot = slot + 1 == S ? 0 : slot + 1;
            fill = fill + 1 == S ? 0 : fill + 1;
            if (uw >= d.nu) continue;   // the whole warp: columns beyond the detector
            const float fz = (float)iz;
            const int ib = (int)((pu0 + iz * du0) >> 32), jb = (int)((pv0 + iz * dv0) >> 32) & ~3;
            WalkTaps<K>* ut = s_ut[warp];
            float tw[K];
            taps_at<K>(tomo_frac(pu), fmaf(fz, dwx, wx), tw);
            if (UPW == 32 || lane < UPW) store_taps(ut[lane], tw);
            const int row = (int)(pu >> 32) - ib;
            const int before = __shfl_up_sync(0xffffffffu, row, 1);
            const unsigned adv1 = __ballot_sync(0xffffffffu, row > before);
            const unsigned adv2 = K > 2 ? __ballot_sync(0xffffffffu, row > before + 1) : 0u;
            const int first = __shfl_sync(0xffffffffu, row, 0);
            RowWalk<K, NP> rw;
            rw.stride = pcols;
            const float wv = fmaf(fz, dwy, wy);
#pragma unroll
            for (int q = 0; q < NP; q++) {
                float a[K], e[K];
                taps_at<K>(tomo_frac(pv[2 * q]), wv, a);
                taps_at<K>(tomo_frac(pv[2 * q + 1]), wv, e);
#pragma unroll
                for (int k = 0; k < K; k++) rw.t[k][q] = f2_pack(a[k], e[k]);
            }
#pragma unroll
            for (int q = 0; q < 2 * NP; q++)
                rw.next[q] = smem + now * patch + first * pcols + ((int)(pv[q] >> 32) - jb);
            __syncwarp();
            rw.start();
#pragma unroll
            for (int j = 0; j < UPW; j++) {
                if (j > 0) {
                    if ((adv1 >> j) & 1) rw.advance();
                    if (K > 2 && ((adv2 >> j) & 1)) rw.advance();
                }
                add_taps(ut[j], rw, acc[j]);
            }
            pu += du;
#pragma unroll
            for (int q = 0; q < 2 * NP; q++) pv[q] += dv[q];
        }
        cp_async_wait<0>();
        __syncthreads();   // the next view refills the slots
#pragma unroll
        for (int j = 0; j < UPW; j++) {
            const int iu = uw + j;
#pragma unroll
            for (int q = 0; q < 2 * NP; q++) {
                const int iv = v0 + lane + 32 * q;
                if (iu < d.nu && iv < d.nv) {
                    const float2 a = f2_unpack(acc[j][q / 2]);
                    const float u = (iu - d.off_u - (d.nu - 1) / 2.0f) * d.du;
                    const float v = (iv - d.off_v - (d.nv - 1) / 2.0f) * d.dv;
                    prj[(((long long)b * d.nu + iu) * d.nview + view) * d.nv * d.nc + (long long)iv * d.nc + c] =
                        (q & 1 ? a.y : a.x) * (float)tomo_len_weight(dc, sp, u, v, d.dz);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Backprojection on tiles.
//
// The voxel's left face ix falls on the detector at u(ix, z) = au + r(z)
// (bu0 + ix dxu) cells, so voxels cover intervals of width r dxu; the same for
// v along y.
// ---------------------------------------------------------------------------
struct TomoBpGeo {
    double au, bu0, dxu, av, bv0, dyv;
    double zs, num;   // r(iz) = num / (z(iz) - zs)
};
__device__ __forceinline__ TomoBpGeo tomo_bp_geo(const TomoDims& d, const float* dc, const float* sp) {
    TomoBpGeo g;
    g.au = ((double)sp[0] - dc[0]) / d.du + d.off_u + (d.nu - 1) / 2.0;
    g.av = ((double)sp[1] - dc[1]) / d.dv + d.off_v + (d.nv - 1) / 2.0;
    g.dxu = (double)d.dx / d.du;
    g.dyv = (double)d.dy / d.dv;
    g.bu0 = ((double)d.cx - sp[0]) / d.du - (d.nx / 2.0) * g.dxu;
    g.bv0 = ((double)d.cy - sp[1]) / d.dv - (d.ny / 2.0) * g.dyv;
    g.zs = sp[2];
    g.num = (double)dc[2] - sp[2];
    return g;
}
__device__ __forceinline__ double tomo_bp_r(const TomoDims& d, const TomoBpGeo& g, int iz) {
    return g.num / ((iz - (d.nz - 1) / 2.0) * d.dz + d.cz - g.zs);
}

// Tile of a block of 4 warps: 4 xpw x 32 ypl x tz voxels.
template <int K>
struct TomoBpTile;
template <>
struct TomoBpTile<3> {
    static constexpr int xpw = 8, ypl = 2, tz = 4;
};
template <>
struct TomoBpTile<4> {
    static constexpr int xpw = 4, ypl = 2, tz = 4;
};
constexpr int kTomoBpSmem = 69 * 1024;   // with the static tables, three blocks per SM

// Patch of detector cells under a tile in any place of the grid: rows (u) and
// columns (v, a multiple of 4); rlo, rhi bound r, step |r(iz + 1) - r(iz)|.
template <int K>
__device__ __forceinline__ int2 tomo_bp_patch(const TomoDims& d, const TomoBpGeo& g, double rhi, double step) {
    using Tl = TomoBpTile<K>;
    const double bu = fmax(fabs(g.bu0), fabs(fma((double)(d.nx + 4 * Tl::xpw), g.dxu, g.bu0)));
    const double bv = fmax(fabs(g.bv0), fabs(fma((double)(d.ny + 32 * Tl::ypl), g.dyv, g.bv0)));
    const double rows = 4 * Tl::xpw * rhi * g.dxu + (Tl::tz - 1) * step * bu;
    const double cols = 32 * Tl::ypl * rhi * g.dyv + (Tl::tz - 1) * step * bv;
    if (!(rows < 4096 && cols < 4096)) return make_int2(1 << 15, 1 << 15);
    return make_int2((int)rows + K + 2, ((int)(cols + 2e-3) + K + 2 + 6) & ~3);
}

// How many cells a voxel's footprint can touch per axis in this view: 3 (at
// most 2 cells wide), 4 (at most 3), or 0 where the tile kernel does not apply;
// its patch, in floats, for either kernel's tile.
__device__ __forceinline__ int tomo_bp_class(const TomoDims& d, const float* dc, const float* sp, int& patch3, int& patch4) {
    const TomoBpGeo g = tomo_bp_geo(d, dc, sp);
    const double r0 = tomo_bp_r(d, g, 0), r1 = tomo_bp_r(d, g, d.nz - 1);
    const double rlo = fmin(r0, r1), rhi = fmax(r0, r1);
    const double lo = rlo * fmin(g.dxu, g.dyv), hi = rhi * fmax(g.dxu, g.dyv);
    // r > 0 at both ends and monotone in between: the source is not between the planes
    if (!(lo > 1e-3 && hi <= 3.0)) return 0;
    if (!((-(d.nz - 1) / 2.0 * d.dz + d.cz - g.zs) * ((d.nz - 1) / 2.0 * d.dz + d.cz - g.zs) > 0)) return 0;
    const double ue = fmax(fabs(g.bu0), fabs(fma((double)(d.nx + 64), g.dxu, g.bu0))) * rhi + fabs(g.au);
    const double ve = fmax(fabs(g.bv0), fabs(fma((double)(d.ny + 64), g.dyv, g.bv0))) * rhi + fabs(g.av);
    if (!(ue < 1e6 && ve < 1e6)) return 0;
    const double step = d.nz < 2 ? 0.0
                                 : fmax(fabs(tomo_bp_r(d, g, 1) - r0), fabs(r1 - tomo_bp_r(d, g, d.nz - 2)));
    const int2 p3 = tomo_bp_patch<3>(d, g, rhi, step), p4 = tomo_bp_patch<4>(d, g, rhi, step);
    patch3 = p3.x * p3.y;
    patch4 = p4.x * p4.y;
    return hi <= 2.0 ? 3 : 4;
}

// The class of the whole call: 0 if some view has class 0 or a patch that does not
// fit twice, else the largest (a class's kernel also serves the narrower footprints,
// on its own tile), in the word's low byte; above it the largest patch in floats.
__global__ void __launch_bounds__(128) tomo_bp_decide(double* sat, const float* __restrict__ detCenter,
                                                      const float* __restrict__ src, TomoDims d) {
    __shared__ int s_patch[2];
    if (threadIdx.x < 2) s_patch[threadIdx.x] = 0;
    __syncthreads();
    int found = 0;   // bit k: a view of class k
    for (int v = threadIdx.x; v < d.nview; v += 128) {
        int p3 = 0, p4 = 0;
        found |= 1 << tomo_bp_class(d, detCenter + 3 * v, src + 3 * v, p3, p4);
        atomicMax(&s_patch[0], p3);
        atomicMax(&s_patch[1], p4);
    }
    const bool any0 = __syncthreads_or(found & 1) != 0, four = __syncthreads_or(found & 16) != 0;
    const long long patch = s_patch[four];
    if (threadIdx.x == 0)
        *reinterpret_cast<unsigned long long*>(sat) =
            any0 || patch * 8 > kTomoBpSmem ? 0ull : (unsigned long long)(patch << 8 | (four ? 4 : 3));
}

// Length-weighted projections of one (b, c) in rows of v, wp[view][u][pitch]
// (pitch = nv rounded up to 4, the padding zero), the magnifications
// rt[view][iz] and the views' {au, bu0, av, bv0} geo[view][4].  A thread weights
// kTomoWeightRows cells along u in FP64, sharing the view's division.  Block 256
// along v; blockIdx = (v, u / kTomoWeightRows, view).
constexpr int kTomoWeightRows = 8;
__global__ void __launch_bounds__(256) tomo_weight_kernel(float* __restrict__ wp, double* __restrict__ rt,
                                                          double* __restrict__ geo, const double* sat,
                                                          const float* __restrict__ prj,
                                                          const float* __restrict__ detCenter,
                                                          const float* __restrict__ src, TomoDims d, int pitch, int b,
                                                          int c, int weight_all) {
    if (tomo_word(sat) == 0) return;
    const int view = blockIdx.z, u0 = blockIdx.y * kTomoWeightRows, iv = blockIdx.x * 256 + threadIdx.x;
    const float* dc = detCenter + 3 * view;
    const float* sp = src + 3 * view;
    if (u0 == 0 && blockIdx.x == 0) {
        const TomoBpGeo g = tomo_bp_geo(d, dc, sp);
        for (int iz = threadIdx.x; iz < d.nz; iz += 256) rt[(long long)view * d.nz + iz] = tomo_bp_r(d, g, iz);
        if (threadIdx.x == 0) {
            geo[4 * view] = g.au;
            geo[4 * view + 1] = g.bu0;
            geo[4 * view + 2] = g.av;
            geo[4 * view + 3] = g.bv0;
        }
    }
    if (iv >= pitch) return;
    float val[kTomoWeightRows];
#pragma unroll
    for (int k = 0; k < kTomoWeightRows; k++) {
        const int iu = u0 + k;
        val[k] = iv < d.nv && iu < d.nu ? __ldg(prj + (((long long)b * d.nu + iu) * d.nview + view) * d.nv * d.nc +
                                                (long long)iv * d.nc + c)
                                        : 0.f;
    }
    if (weight_all || view == 0) {
        // tomo_len_weight with the cell-independent parts out of the loop
        const float v = (iv - d.off_v - (d.nv - 1) / 2.0f) * d.dv;
        const double ddz = (double)sp[2] - dc[2], ddy = (double)sp[1] - (dc[1] + v);
        const double scale = (double)d.dz / fabs(ddz), yz = ddy * ddy + ddz * ddz;
#pragma unroll
        for (int k = 0; k < kTomoWeightRows; k++) {
            const float u = (u0 + k - d.off_u - (d.nu - 1) / 2.0f) * d.du;
            const double ddx = (double)sp[0] - (dc[0] + u);
            val[k] = (float)((double)val[k] * (scale * sqrt(fma(ddx, ddx, yz))));
        }
    }
#pragma unroll
    for (int k = 0; k < kTomoWeightRows; k++)
        if (u0 + k < d.nu) wp[((long long)view * d.nu + u0 + k) * pitch + iv] = val[k];
}

// A block owns a tile of voxels and walks the views; the patch of detector
// cells under the tile arrives in shared memory one view ahead or more.  As in
// tomo_fp_tile_kernel, a lane keeps the taps of its rows y along v, the taps
// along u of the warp's XPW columns and TZ planes come from one lane each, and
// a warp walks its columns with the v-weighted sums of the K cell rows under
// the current one.  The TZ planes share one patch (they see nearly the same
// cells), which cuts the patch traffic from L2 by as much, and their voxels are
// stored together.  Positions are FP64 at the lanes' first row and column and
// FP32 offsets from the patch's corner beyond (under 200 cells, so good to
// ~1e-5 cells).  Bound by instruction issue.  512x512x128 voxels, 736x736
// cells, 25 views: 1.40 ms, where the summed-area-table kernel takes 2.53 ms.
template <int K>
__global__ void __launch_bounds__(128, 3)
    tomo_bp_tile_kernel(float* __restrict__ img, const float* __restrict__ wp, const double* __restrict__ rt,
                        const double* __restrict__ geo, const double* sat, TomoDims d, int pitch, int b, int c) {
    constexpr int XPW = TomoBpTile<K>::xpw, NP = TomoBpTile<K>::ypl / 2, TZ = TomoBpTile<K>::tz;
    constexpr int TX = 4 * XPW, TY = 64 * NP;
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(16) WalkTaps<K> s_ut[4][XPW * TZ];   // per warp; rewritten after the next barrier
    __shared__ int4 s_win[4];   // per slot: first u, first v (a multiple of 4), columns (a multiple of 4)
    const unsigned long long word = tomo_word(sat);
    if ((word & 255) != K) return;
    const int patch = (int)(word >> 8);
    const int S = min(4, kTomoBpSmem / (4 * patch));   // >= 2
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ntx = (d.nx + TX - 1) / TX, nty = (d.ny + TY - 1) / TY, ntz = (d.nz + TZ - 1) / TZ;
    const double dxu = (double)d.dx / d.du, dyv = (double)d.dy / d.dv;
    // tiles with z fastest: the blocks resident at a time cover few (x, y)
    // columns, whose patches in all views stay in L2
    for (int tile = blockIdx.x; tile < ntx * nty * ntz; tile += gridDim.x) {
        const int z0 = (tile % ntz) * TZ, x0 = (tile / ntz % ntx) * TX, y0 = (tile / ntz / ntx) * TY;
        const int xw = x0 + warp * XPW;
        const int z1 = min(z0 + TZ, d.nz) - 1;
        auto issue = [&](int view, int slot) {
            // u and v of the tile's corners: r is monotone along z
            const double ra = __ldg(rt + (long long)view * d.nz + z0), rb = __ldg(rt + (long long)view * d.nz + z1);
            const double au = __ldg(geo + 4 * view), bu0 = __ldg(geo + 4 * view + 1);
            const double av = __ldg(geo + 4 * view + 2), bv0 = __ldg(geo + 4 * view + 3);
            const double xa = fma((double)x0, dxu, bu0), xb = fma((double)(x0 + TX - 1), dxu, bu0);
            const double ya = fma((double)y0, dyv, bv0), yb = fma((double)(y0 + TY - 1), dyv, bv0);
            const int ub = (int)floor(fmin(fma(ra, xa, au), fma(rb, xa, au)));
            const int vb = (int)floor(fmin(fma(ra, ya, av), fma(rb, ya, av)) - 1e-3) & ~3;
            const int rows = (int)floor(fmax(fma(ra, xb, au), fma(rb, xb, au))) - ub + K;
            const int cols = ((int)floor(fmax(fma(ra, yb, av), fma(rb, yb, av)) + 1e-3) - vb + K + 3) & ~3;
            if (threadIdx.x == 0) s_win[slot] = make_int4(ub, vb, cols, 0);
            const int j = vb + 4 * lane;
            const float* row = wp + ((long long)view * d.nu + ub + warp) * pitch + j;
            const uint32_t dst = smem_u32(smem + slot * patch) + (warp * cols + 4 * lane) * 4;
            for (int q = 0; q < cols; q += 128) {
                if (4 * lane + q >= cols) break;
                const bool jin = j + q >= 0 && j + q < pitch;
                const float* s = row + q;
                uint32_t t = dst + 4 * q;
#pragma unroll 4
                for (int r = warp; r < rows; r += 4) {
                    const bool in = jin && (unsigned)(ub + r) < (unsigned)d.nu;
                    cp_async16(t, in ? s : wp, in);
                    s += 4 * pitch;
                    t += 16 * cols;
                }
            }
        };
        f32x2 acc[TZ][XPW][NP];
#pragma unroll
        for (int z = 0; z < TZ; z++)
#pragma unroll
            for (int k = 0; k < XPW; k++)
#pragma unroll
                for (int q = 0; q < NP; q++) acc[z][k][q] = 0ull;
        for (int s = 0; s < S - 1; s++) {
            if (s < d.nview) issue(s, s);
            cp_async_commit();
        }
        int slot = 0, fill = S - 1;
        for (int view = 0; view < d.nview; view++) {
            if (S == 2) cp_async_wait<0>();
            else if (S == 3) cp_async_wait<1>();
            else cp_async_wait<2>();
            __syncthreads();   // this view's patch is in; every warp has left the slot filled next
            if (view + S - 1 < d.nview) issue(view + S - 1, fill);
            cp_async_commit();
            const int ub = s_win[slot].x, vb = s_win[slot].y, cols = s_win[slot].z;
            const double au = __ldg(geo + 4 * view), bu0 = __ldg(geo + 4 * view + 1);
            const double av = __ldg(geo + 4 * view + 2), bv0 = __ldg(geo + 4 * view + 3);
            WalkTaps<K>* ut = s_ut[warp];
            // lane = plane * XPW + column
            const int zi = lane / XPW % TZ;
            const double rz = __ldg(rt + (long long)view * d.nz + min(z0 + zi, d.nz - 1));
            const double ul = fma(rz, fma((double)(xw + lane % XPW), dxu, bu0), au);
            const double uf = floor(ul);
            float tw[K];
            taps_at<K>((float)(ul - uf), (float)(rz * dxu), tw);
            if (lane < XPW * TZ) store_taps(ut[lane], tw);
            const int urow = (int)uf - ub;
            const int before = __shfl_up_sync(0xffffffffu, urow, 1);
            const unsigned adv1 = __ballot_sync(0xffffffffu, urow > before);
            const unsigned adv2 = __ballot_sync(0xffffffffu, urow > before + 1);
            const unsigned adv3 = K > 3 ? __ballot_sync(0xffffffffu, urow > before + 2) : 0u;
            // v of row y0 from the patch's first column, and the step per row
            const float vstart = (float)(fma(rz, fma((double)y0, dyv, bv0), av) - vb), vstep = (float)(rz * dyv);
            __syncwarp();
#pragma unroll
            for (int z = 0; z < TZ; z++) {
                const float va = __shfl_sync(0xffffffffu, vstart, z * XPW);
                const float vs = __shfl_sync(0xffffffffu, vstep, z * XPW);
                const int first = __shfl_sync(0xffffffffu, urow, z * XPW);
                RowWalk<K, NP> rw;
                rw.stride = cols;
#pragma unroll
                for (int q = 0; q < NP; q++) {
                    float t[2][K];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const float v = fmaf((float)(lane + 64 * q + 32 * h), vs, va);
                        const float y = __fadd_rd(v, 12582912.0f);   // floor, 0 <= v < 2^22
                        taps_at<K>(v - (y - 12582912.0f), vs, t[h]);
                        rw.next[2 * q + h] = smem + slot * patch + first * cols + (__float_as_int(y) - 0x4B400000);
                    }
#pragma unroll
                    for (int k = 0; k < K; k++) rw.t[k][q] = f2_pack(t[0][k], t[1][k]);
                }
                rw.start();
#pragma unroll
                for (int j = 0; j < XPW; j++) {
                    if (j > 0) {
                        if ((adv1 >> (z * XPW + j)) & 1) rw.advance();
                        if ((adv2 >> (z * XPW + j)) & 1) rw.advance();
                        if (K > 3 && ((adv3 >> (z * XPW + j)) & 1)) rw.advance();
                    }
                    add_taps(ut[z * XPW + j], rw, acc[z][j]);
                }
            }
            slot = slot + 1 == S ? 0 : slot + 1;
            fill = fill + 1 == S ? 0 : fill + 1;
        }
        cp_async_wait<0>();
        __syncthreads();   // the next tile refills the slots
#pragma unroll
        for (int j = 0; j < XPW; j++)
#pragma unroll
            for (int q = 0; q < 2 * NP; q++) {
                const int ix = xw + j, iy = y0 + lane + 32 * q;
                if (ix < d.nx && iy < d.ny) {
                    float v[TZ];
#pragma unroll
                    for (int z = 0; z < TZ; z++) {
                        const float2 a = f2_unpack(acc[z][j][q / 2]);
                        v[z] = q & 1 ? a.y : a.x;
                    }
                    float* out = img + ((((long long)b * d.nx + ix) * d.ny + iy) * d.nz + z0) * d.nc + c;
                    if (d.nc == 1 && z0 + TZ <= d.nz && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
                        *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
                    } else {
#pragma unroll
                        for (int z = 0; z < TZ; z++)
                            if (z0 + z < d.nz) out[(long long)z * d.nc] = v[z];
                    }
                }
            }
    }
}

// ---------------------------------------------------------------------------
// Table kernels: the calls and views that the tiles leave out.  Whether a call needs
// them they read in its word, so their grids are no larger than the GPU holds and
// walk their work.  (Blocks per SM are bounded from below because the compiler
// otherwise trades them for registers: with two instead of four the backprojection
// of 300 x 300 x 64 voxels from 25 views took 527 us, 457 now, 436 with a block per
// tile and no word to read; the forward projection of 25 views of 400 x 400 cells takes
// 1065 with eight, and took 774 with a block per 31 x 4 cells and neither word nor
// classes to read, which as many blocks cost every other call.)
//
// Tables (FP64).  FP: per z plane, row prefixes along x of image row y,
// layout [z][y + 1][x] (x fastest, x in [0, nx]); a rectangle integral is the
// sum over the rows it overlaps (rows_integral), which equals the reference's
// summed-area-table corner form.  BP: per view, row prefixes along u of the
// length-weighted projections, layout [view][v + 1][u] (u fastest, u in
// [0, nu]), then summed along v in place (tomo_bp_sat_v) into the (u, v)
// summed-area table.  Rows run along the axis that the lanes of the main
// kernels walk, so their reads are coalesced.
// Row prefixes are built by a tiled pass that reads the source along its
// contiguous axis, transposes 32 x 32 tiles through shared memory and scans
// along the row with warp scans (carry across tiles).
// ---------------------------------------------------------------------------

// Row prefixes R[z][y + 1][x + 1] = sum_{x' <= x} img[x'][y][z].  Block
// (32, 8): blockIdx.x = y, blockIdx.y = a tile of 32 planes.
// `tiled`: only if the call's word (left as it is, a zero) asks for the tables.
__global__ void __launch_bounds__(256) tomo_sat_x(double* __restrict__ sat, const float* __restrict__ img, TomoDims d,
                                                  int tiled, int b, int c) {
    if (tiled && (tomo_word(sat) & ~kTomoMixed)) return;
    __shared__ float tile[32][33];
    const int y = blockIdx.x, z0 = blockIdx.y * 32;
    const int lane = threadIdx.x, w = threadIdx.y;
    const long long plane = (long long)(d.nx + 1) * (d.ny + 1), row = d.nx + 1;
    const long long sx = (long long)d.ny * d.nz * d.nc;   // img stride along x
    const float* base = img + (long long)b * d.nx * sx + (long long)y * d.nz * d.nc + c;
    double carry[4] = {0.0, 0.0, 0.0, 0.0};
    for (int x0 = 0; x0 < d.nx; x0 += 32) {
#pragma unroll
        for (int k = 0; k < 4; k++) {   // rows x0 + w + 8k, lanes along z (contiguous)
            const int x = x0 + w + 8 * k, z = z0 + lane;
            tile[w + 8 * k][lane] = (x < d.nx && z < d.nz) ? base[(long long)x * sx + (long long)z * d.nc] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; k++) {   // plane z0 + w + 8k, lanes along x
            const int zz = w + 8 * k, z = z0 + zz;
            const double v = (double)tile[lane][zz];
            const double incl = warp_incl_scan(v);
            if (z < d.nz && x0 + lane < d.nx) sat[z * plane + (y + 1) * row + (x0 + lane + 1)] = carry[k] + incl;
            carry[k] += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncthreads();
    }
    // column x = 0 of row y + 1, and row y = 0 of the tile's planes
    const int z = z0 + lane;
    if (w == 0 && z < d.nz) sat[z * plane + (y + 1) * row] = 0.0;
    if (y == 0)
        for (int zz = w; zz < 32 && z0 + zz < d.nz; zz += 8)
            for (int x = lane; x <= d.nx; x += 32)
                if (!tiled || z0 + zz > 0 || x > 0) sat[(z0 + zz) * plane + x] = 0.0;
}

// Weighted row prefixes R[view][v + 1][u + 1] = sum_{u' <= u} w p(u', v).
// weight_all = 0 applies the length weight to view 0 only, as the reference's
// pre-weight launch does (its grid has one row of views,
// DistanceDriven3D.cu:612-621); 1 weights every view.  Block (32, 8):
// blockIdx.x = a tile of 32 detector rows v, blockIdx.y = view.
__global__ void __launch_bounds__(256) tomo_bp_sat_u(double* __restrict__ sat, const float* __restrict__ prj,
                                                     const float* __restrict__ detCenter,
                                                     const float* __restrict__ src, TomoDims d, int b, int c,
                                                     int weight_all, int tiled) {
    if (tiled && tomo_word(sat)) return;
    __shared__ double tile[32][33];
    const int v0 = blockIdx.x * 32, view = blockIdx.y;
    const int lane = threadIdx.x, w = threadIdx.y;
    const float* dc = detCenter + 3 * view;
    const float* sp = src + 3 * view;
    const bool weighted = weight_all || view == 0;
    const long long vplane = (long long)(d.nu + 1) * (d.nv + 1), row = d.nu + 1;
    double* S = sat + view * vplane;
    const long long su = (long long)d.nview * d.nv * d.nc;   // prj stride along u
    const float* base = prj + (long long)b * d.nu * su + (long long)view * d.nv * d.nc + c;
    double carry[4] = {0.0, 0.0, 0.0, 0.0};
    for (int u0 = 0; u0 < d.nu; u0 += 32) {
#pragma unroll
        for (int k = 0; k < 4; k++) {   // cells u0 + w + 8k, lanes along v (contiguous)
            const int iu = u0 + w + 8 * k, iv = v0 + lane;
            double val = 0.0;
            if (iu < d.nu && iv < d.nv) {
                val = (double)base[(long long)iu * su + (long long)iv * d.nc];
                if (weighted) {
                    const float u = (iu - d.off_u - (d.nu - 1) / 2.0f) * d.du;
                    const float v = (iv - d.off_v - (d.nv - 1) / 2.0f) * d.dv;
                    val *= tomo_len_weight(dc, sp, u, v, d.dz);
                }
            }
            tile[w + 8 * k][lane] = val;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; k++) {   // row v0 + w + 8k, lanes along u
            const int vv = w + 8 * k, iv = v0 + vv;
            const double incl = warp_incl_scan(tile[lane][vv]);
            if (iv < d.nv && u0 + lane < d.nu) S[(iv + 1) * row + (u0 + lane + 1)] = carry[k] + incl;
            carry[k] += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncthreads();
    }
    const int iv = v0 + lane;
    if (w == 0 && iv < d.nv) S[(iv + 1) * row] = 0.0;
    if (blockIdx.x == 0)
        for (int u = lane + 32 * w; u <= d.nu; u += 256) S[u] = 0.0;
}

// In place along v: T[view][k][u] = sum_{k' <= k} R[view][k'][u], the (u, v)
// summed-area table of the weighted projections (row 0 stays 0), the
// quantity of the reference's AccumulateUVAlongVKernel (DistanceDriven3D.cu:459-475).
// A warp scans 32 u columns (lanes along u, coalesced) down all rows, loading
// 8 rows ahead of the running sum.  `tiled`: the tile kernels have run and
// this one only serves the calls whose class they leave out (likewise
// tomo_bp_sat_u and tomo_bp_kernel).  Block (32, 4): blockIdx.x * 4 + warp = a
// strip of 32 columns, blockIdx.y = view.
__global__ void __launch_bounds__(128) tomo_bp_sat_v(double* __restrict__ sat, TomoDims d, int tiled) {
    if (tiled && tomo_word(sat)) return;
    const int u = (blockIdx.x * 4 + threadIdx.y) * 32 + threadIdx.x;
    // the two pad entries after the last view's table (read with weight 0
    // by the backprojection's u + 1 neighbour at u = nu)
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.y == 0 && threadIdx.x < 2)
        sat[(long long)d.nview * (d.nu + 1) * (d.nv + 1) + threadIdx.x] = 0.0;
    if (u > d.nu) return;
    const long long row = d.nu + 1;
    double* T = sat + (long long)blockIdx.y * row * (d.nv + 1) + u;
    double acc = 0.0;
    for (int k0 = 1; k0 <= d.nv; k0 += 8) {
        double v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = k0 + i <= d.nv ? T[(k0 + i) * row] : 0.0;
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (k0 + i <= d.nv) {
                acc += v[i];
                T[(k0 + i) * row] = acc;
            }
    }
}

// Clamp_float + the index / weight of one coordinate of InterpolateXY /
// InterpolateUV (DistanceDriven3D.cu:75-135, :493-517) on a grid of n points.
struct Lerp {
    int i0, i1;
    double w;
};
// The index and the fraction come from a round-down add against 1.5 * 2^23
// (exact for 0 <= x < 2^22) instead of conversions on the XU pipe; a NaN
// coordinate clamps to 0.
__device__ __forceinline__ Lerp lerp_at(float x, int n) {
    x = fminf(fmaxf(x, 0.f), (float)(n - 1));
    const float y = __fadd_rd(x, 12582912.0f);
    Lerp l;
    l.i0 = __float_as_int(y) - 0x4B400000;
    l.i1 = min(l.i0 + 1, n - 1);
    l.w = (double)(x - (y - 12582912.0f));
    return l;
}
// Integral over [y1, y2] (clamped to [0, n]; the result changes sign when
// y2 < y1) of the row prefixes of a table R[row j + 1][col], interpolated
// linearly at the column lc: the summed-area-table difference S(c, y2) -
// S(c, y1) written as the rows that [y1, y2] overlaps, each weighted by its
// overlap.  Equal to the bilinear corner form of InterpolateXY / UV in exact
// arithmetic, with one or two rows instead of four corner reads.
__device__ __forceinline__ double rows_integral(const double* __restrict__ R, const Lerp& lc, float y1, float y2, int n,
                                                long long row) {
    float lo = fminf(y1, y2), hi = fmaxf(y1, y2);
    lo = fminf(fmaxf(lo, 0.f), (float)n);
    hi = fminf(fmaxf(hi, 0.f), (float)n);
    double acc = 0.0;
    // rows j < n overlapped by [lo, hi]; j and its float value fj from a
    // round-down add, as in lerp_at
    const float y = __fadd_rd(lo, 12582912.0f);
    float fj = y - 12582912.0f;
    const double* r = R + (long long)(__float_as_int(y) - 0x4B400000 + 1) * row;
#pragma unroll 4
    for (; fj < hi; fj += 1.f, r += row) {
        const float ov = fminf(hi, fj + 1.f) - fmaxf(lo, fj);
        acc += (r[lc.i0] * (1 - lc.w) + r[lc.i1] * lc.w) * (double)ov;
    }
    return y2 >= y1 ? acc : -acc;
}

// FP: lane i of a warp owns detector column iu = 31 blockIdx.x + i and its
// left cell edge; lane 31 only supplies the right edge of lane 30's cell.  A
// warp handles one detector row v of one view, and per z plane each lane
// evaluates D = S(x_e, y2) - S(x_e, y1) at its edge from the rows [y1, y2]
// overlaps, so the rectangle integral of a cell is D(next lane) - D(this
// lane): two reads per overlapped row instead of the reference's 16 corner
// reads.  The rectangle's area is (x_{e+1} - x_e)(y2 - y1) = drx dry
// (z - sz)^2, exact for the straight edge rays.
__global__ void __launch_bounds__(128, 8) tomo_fp_kernel(float* __restrict__ prj, const double* __restrict__ sat,
                                                      const float* __restrict__ detCenter,
                                                      const float* __restrict__ src, TomoDims d, int tiled, int b,
                                                      int c) {
    const unsigned long long word = tiled ? tomo_word(sat) : 0ull;
    if (word & ~kTomoMixed) return;
    const int lane = threadIdx.x;
    const int nut = (d.nu + 30) / 31, nvt = (d.nv + blockDim.y - 1) / blockDim.y;
    for (long long job = blockIdx.x; job < (long long)nut * nvt * d.nview; job += gridDim.x) {
        const int iview = (int)(job / (nut * nvt)), item = (int)(job - (long long)iview * (nut * nvt));
        const float* dc = detCenter + 3 * iview;
        const float* sp = src + 3 * iview;
        if (word && tomo_fp_class(d, dc, sp) != 0) continue;   // a call that has tiled views too
        const int iu = (item % nut) * 31 + lane;
        const int iv = (item / nut) * blockDim.y + threadIdx.y;
        if (iv >= d.nv) continue;   // warp-uniform
        const float u = (iu - d.off_u - (d.nu - 1) / 2.0f) * d.du;
        const float v = (iv - d.off_v - (d.nv - 1) / 2.0f) * d.dv;
        auto img_x = [&](float px) { return (px - d.cx) / d.dx + d.nx / 2.0f; };
        auto img_y = [&](float py) { return (py - d.cy) / d.dy + d.ny / 2.0f; };
        auto img_z = [&](float pz) { return (pz - d.cz) / d.dz + d.nz / 2.0f; };
        const float sx = img_x(sp[0]), sy = img_y(sp[1]), sz = img_z(sp[2]);
        const float zd = img_z(dc[2]);
        const float xe = img_x(dc[0] + u - d.du / 2);
        const float ya = img_y(dc[1] + v - d.dv / 2), yb = img_y(dc[1] + v + d.dv / 2);
        const float rxe = (xe - sx) / (zd - sz);
        const float rya = (ya - sy) / (zd - sz), ryb = (yb - sy) / (zd - sz);
        const float drx = __shfl_down_sync(0xffffffffu, rxe, 1) - rxe;   // signed, as are D and dry
        const float k = 1.0f / (drx * (ryb - rya));
        const long long plane = (long long)(d.nx + 1) * (d.ny + 1), row = d.nx + 1;
        float val = 0.f;
        for (int iz = 0; iz < d.nz; iz++) {
            const float t = (float)iz - sz;
            const Lerp lx = lerp_at(sx + rxe * t, d.nx + 1);
            const double D = rows_integral(sat + iz * plane, lx, sy + rya * t, sy + ryb * t, d.ny, row);
            const double q = __shfl_down_sync(0xffffffffu, D, 1) - D;
            val = fmaf((float)q, __fdividef(k, t * t), val);
        }
        if (lane < 31 && iu < d.nu) {
            val *= (float)tomo_len_weight(dc, sp, u, v, d.dz);
            prj[(long long)b * d.nu * d.nview * d.nv * d.nc + ((long long)iu * d.nview + iview) * d.nv * d.nc +
                (long long)iv * d.nc + c] = val;
        }
    }
}

// BP: lane i of a warp owns voxel column ix = 31 blockIdx.y + i and its left
// face; lane 31 only supplies the right face of lane 30's voxel.  A warp
// handles kTomoBpRows consecutive voxels y0 .. y0 + 7 of one z plane.  Per
// view each lane evaluates the (u, v) summed-area table T of the weighted
// projections, bilinearly (InterpolateUV, DistanceDriven3D.cu:493-517), at
// its face's detector coordinate u_e (ProjectConeToDetCart, :478-489) and the
// detector coordinates f_0 .. f_8 of the 8 voxels' v faces (the same for
// every lane of the warp): D_j = T(u_e, f_(j+1)) - T(u_e, f_j), and the
// voxel's rectangle integral is D_j(next lane) - D_j(this lane), divided by
// its area r^2 dx dy / (du dv).  The reference reads 4 corners of 4 bilinear
// samples per voxel and view; sharing corners between neighbouring voxels
// in x (shuffles) and in y (the face between them) leaves 4 table reads per
// voxel and view, all independent of one another.
constexpr int kTomoBpRows = 8;

__global__ void __launch_bounds__(256, 4) tomo_bp_kernel(float* __restrict__ img, const double* __restrict__ sat,
                                                      const float* __restrict__ detCenter,
                                                      const float* __restrict__ src, TomoDims d, int b, int c,
                                                      int tiled) {
    if (tiled && tomo_word(sat)) return;
    // z runs fastest over the grid, so the CTAs resident at a time cover few
    // (x, y) columns and their detector footprints in all views stay in L2
    const int lane = threadIdx.x;
    const int ntx = (d.nx + 30) / 31, nty = (d.ny + blockDim.y * kTomoBpRows - 1) / (blockDim.y * kTomoBpRows);
    for (int tile = blockIdx.x; tile < d.nz * ntx * nty; tile += gridDim.x) {
        const int iz = tile % d.nz;
        const int ix = (tile / d.nz % ntx) * 31 + lane;
        const int y0 = ((tile / d.nz / ntx) * blockDim.y + threadIdx.y) * kTomoBpRows;
        if (y0 >= d.ny) continue;   // warp-uniform
        const int ny_w = min(kTomoBpRows, d.ny - y0);
        const float xf = (ix - (d.nx - 1) / 2.0f) * d.dx + d.cx - d.dx / 2;
        const float yb = (y0 - (d.ny - 1) / 2.0f) * d.dy + d.cy - d.dy / 2;   // lower face of voxel y0
        const float z = (iz - (d.nz - 1) / 2.0f) * d.dz + d.cz;
        const float cu = d.off_u + (d.nu - 1) / 2.0f, cv = d.off_v + (d.nv - 1) / 2.0f;
        const float aunit = d.dx * d.dy / (d.du * d.dv);
        const float idu = 1.0f / d.du, idv = 1.0f / d.dv;
        const long long vplane = (long long)(d.nu + 1) * (d.nv + 1);
        const int row = d.nu + 1;
        float acc[kTomoBpRows];
    #pragma unroll
        for (int j = 0; j < kTomoBpRows; j++) acc[j] = 0.f;
#pragma unroll 2
        for (int view = 0; view < d.nview; view++) {
            const float* dc = detCenter + 3 * view;
            const float* sp = src + 3 * view;
            const float r = (dc[2] - sp[2]) / (z - sp[2]);
            const float ue = fmaf(sp[0] - dc[0] + r * (xf - sp[0]), idu, cu);
            const float ov0 = sp[1] - dc[1], wgt = __fdividef(1.0f, r * r * aunit);
            // u_e clamped to [0, nu]: column iu and its neighbour iu + 1 with
            // weight wu (at u_e = nu the neighbour is the next row's zero column
            // or a pad entry, with weight 0)
            const float uc = fminf(fmaxf(ue, 0.f), (float)d.nu);
            const float uy = __fadd_rd(uc, 12582912.0f);
            const double wu = (double)(uc - (uy - 12582912.0f)), wu1 = 1.0 - wu;
            const double* Tu = sat + view * vplane + (__float_as_int(uy) - 0x4B400000);
            // T(u_e, f_j) at the lower face of voxel y0 + j, from table rows k0
            // and k1 = k0 + 1 (clamped); a face whose k0 is the previous face's
            // k1 (the row index is the same for the whole warp) reuses that row
            int kp = -1;
            double ep = 0.0;
            auto tface = [&](int j) {
                const float f = fmaf(ov0 + r * (fmaf((float)j, d.dy, yb) - sp[1]), idv, cv);
                const Lerp lv = lerp_at(f, d.nv + 1);
                double a;
                if (lv.i0 == kp) {
                    a = ep;
                } else {
                    const double* t0 = Tu + lv.i0 * row;
                    a = t0[0] * wu1 + t0[1] * wu;
                }
                const double* t1 = Tu + lv.i1 * row;
                const double e = t1[0] * wu1 + t1[1] * wu;
                kp = lv.i1;
                ep = e;
                return fma(e - a, lv.w, a);
            };
            double tprev = tface(0);
    #pragma unroll
            for (int j = 0; j < kTomoBpRows; j++) {
                if (j < ny_w) {   // warp-uniform
                    const double t = tface(j + 1);
                    const double D = t - tprev;
                    const double q = __shfl_down_sync(0xffffffffu, D, 1) - D;
                    acc[j] = fmaf((float)q, wgt, acc[j]);
                    tprev = t;
                }
            }
        }
        if (lane < 31 && ix < d.nx) {
            float* out = img + (long long)b * d.nx * d.ny * d.nz * d.nc + (((long long)ix * d.ny + y0) * d.nz + iz) * d.nc + c;
    #pragma unroll
            for (int j = 0; j < kTomoBpRows; j++)
                if (j < ny_w) out[(long long)j * d.nz * d.nc] = acc[j];
        }
    }
}

static int tomo_validate(const TomoDims& d) {
    if (d.nb <= 0 || d.nc <= 0 || d.nx <= 0 || d.ny <= 0 || d.nz <= 0 || d.nu <= 0 || d.nview <= 0 || d.nv <= 0)
        return set_error(RN_ERR_ARG, "tomo: sizes must be positive");
    if (!(d.dx > 0 && d.dy > 0 && d.dz > 0 && d.du > 0 && d.dv > 0))
        return set_error(RN_ERR_ARG, "tomo: pixel and detector sizes must be positive");
    return RN_OK;
}

// The tile kernels' shared memory, once per device.
static std::mutex g_tomo_attr_mu;
static std::vector<char> g_tomo_attr_done;
static int tomo_kernel_attributes() {
    int dev = 0;
    RN_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_tomo_attr_mu);
    if ((int)g_tomo_attr_done.size() <= dev) g_tomo_attr_done.resize(dev + 1, 0);
    if (g_tomo_attr_done[dev]) return RN_OK;
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    RN_CUDA_TRY(cudaFuncSetAttribute(tomo_fp_tile_kernel<2, 16, 2>, attr, kTomoTileSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(tomo_fp_tile_kernel<3, 8, 1>, attr, kTomoTileSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(tomo_bp_tile_kernel<3>, attr, kTomoBpSmem));
    RN_CUDA_TRY(cudaFuncSetAttribute(tomo_bp_tile_kernel<4>, attr, kTomoBpSmem));
    g_tomo_attr_done[dev] = 1;
    return RN_OK;
}

// The scratch's first 16-byte boundary.
static unsigned char* align16(void* p) {
    return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(p) + 15) & ~uintptr_t(15));
}

int tomo_project(float* d_prj, const float* d_img, const float* d_dc, const float* d_src, const TomoDims& d,
                 double* d_sat, cudaStream_t st) {
    RN_TRY(tomo_validate(d));
    RN_TRY(tomo_kernel_attributes());
    // After the call's word the plane-major copy, where the prefix tables of the other
    // views are built afterwards (a volume of a few voxels has no room for it)
    float* vol = reinterpret_cast<float*>(align16(d_sat + 1));
    const int pitch = (d.ny + 3) & ~3;
    const int tiled = 24 + 4 * (size_t)d.nz * d.nx * pitch <= 8 * (size_t)d.nz * (d.nx + 1) * (d.ny + 1);
    // 64 x 128-cell tiles for footprints up to a voxel where they fill the
    // GPU, else 32 x 64-cell tiles for all of them.  What the classes leave to the
    // kernels after the first is not known here: each gets blocks enough to fill the
    // GPU, and its blocks walk the rest of the views, so that one with nothing to do
    // costs little and one with all views is not held up.  (With each cell's views one
    // after another, 60 views of 400 x 400 cells with footprints over a voxel took 2.60
    // ms forward; 0.97 now.)
    const long long big = (long long)((d.nu + 63) / 64) * ((d.nv + 127) / 128) * d.nview;
    const bool use_big = big >= 3 * 148;
    const int views = std::min(d.nview, 65535);
    const long long small = (long long)((d.nu + 31) / 32) * ((d.nv + 63) / 64);
    const long long items = (long long)((d.nu + 30) / 31) * ((d.nv + 3) / 4);
    // grid z: blocks of a view times this are about `want`
    auto fill = [&](long long per_view, long long want) {
        return (unsigned)std::min<long long>(views, (want + per_view - 1) / per_view);
    };
    if (tiled) tomo_fp_decide<<<1, 128, 0, st>>>(d_sat, d_dc, d_src, d);
    for (int b = 0; b < d.nb; b++)
        for (int c = 0; c < d.nc; c++) {
            if (tiled) {
                tomo_planes_kernel<<<dim3((pitch + 31) / 32, (d.nz + 31) / 32, std::min(d.nx, 16)), dim3(32, 8), 0, st>>>(
                    vol, d_img, d_sat, d, pitch, b, c);
                if (use_big)
                    tomo_fp_tile_kernel<2, 16, 2><<<dim3((d.nv + 127) / 128, (d.nu + 63) / 64, views), 128, kTomoTileSmem,
                                                    st>>>(d_prj, vol, d_sat, d_dc, d_src, d, pitch, b, c, 0);
                tomo_fp_tile_kernel<3, 8, 1>
                    <<<dim3((d.nv + 63) / 64, (d.nu + 31) / 32, use_big ? fill(small, 2 * 3 * 148) : views), 128,
                       kTomoTileSmem, st>>>(d_prj, vol, d_sat, d_dc, d_src, d, pitch, b, c, use_big ? 0 : 1);
            }
            tomo_sat_x<<<dim3(d.ny, (d.nz + 31) / 32), dim3(32, 8), 0, st>>>(d_sat, d_img, d, tiled, b, c);
            const unsigned grid = (unsigned)std::min<long long>(items * d.nview, 148 * 16);
            tomo_fp_kernel<<<grid, dim3(32, 4), 0, st>>>(d_prj, d_sat, d_dc, d_src, d, tiled, b, c);
        }
    RN_CUDA_TRY(cudaGetLastError());
    return RN_OK;
}

int tomo_backproject(float* d_img, const float* d_prj, const float* d_dc, const float* d_src, const TomoDims& d,
                     double* d_sat, int weight_all, cudaStream_t st) {
    RN_TRY(tomo_validate(d));
    RN_TRY(tomo_kernel_attributes());
    // after the call's word the weighted projections, then the magnifications, in the
    // scratch of the summed-area tables (too small for them only where a detector of a
    // few cells meets many planes)
    const int pitch = (d.nv + 3) & ~3;
    float* wp = reinterpret_cast<float*>(align16(d_sat + 1));
    const size_t wp_bytes = (size_t)d.nview * d.nu * pitch * sizeof(float);
    double* rt = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(wp) + wp_bytes);
    double* geo = rt + (size_t)d.nview * d.nz;
    const size_t have = ((size_t)d.nview * (d.nu + 1) * (d.nv + 1) + 2) * 8;
    const bool tiled = 24 + wp_bytes + (size_t)d.nview * (d.nz + 4) * 8 <= have && d.nview <= 65535 && d.nu <= 65535;
    auto tiles = [&](int tx, int ty, int tz) {
        const long long n =
            (long long)((d.nx + tx - 1) / tx) * ((d.ny + ty - 1) / ty) * ((d.nz + tz - 1) / tz);
        return (unsigned)std::min<long long>(n, 0x7fffffff);
    };
    if (tiled) tomo_bp_decide<<<1, 128, 0, st>>>(d_sat, d_dc, d_src, d);
    for (int b = 0; b < d.nb; b++)
        for (int c = 0; c < d.nc; c++) {
            if (tiled) {
                tomo_weight_kernel<<<dim3((pitch + 255) / 256, (d.nu + kTomoWeightRows - 1) / kTomoWeightRows, d.nview), 256, 0,
                                     st>>>(
                    wp, rt, geo, d_sat, d_prj, d_dc, d_src, d, pitch, b, c, weight_all);
                tomo_bp_tile_kernel<3><<<tiles(32, 64, 4), 128, kTomoBpSmem, st>>>(d_img, wp, rt, geo, d_sat, d, pitch, b,
                                                                                  c);
                tomo_bp_tile_kernel<4><<<std::min(tiles(16, 64, 4), 148u * 3), 128, kTomoBpSmem, st>>>(
                    d_img, wp, rt, geo, d_sat, d, pitch, b, c);
            }
            tomo_bp_sat_u<<<dim3((d.nv + 31) / 32, d.nview), dim3(32, 8), 0, st>>>(d_sat, d_prj, d_dc, d_src, d, b,
                                                                                    c, weight_all, tiled);
            tomo_bp_sat_v<<<dim3((d.nu + 1 + 127) / 128, d.nview), dim3(32, 4), 0, st>>>(d_sat, d, tiled);
            tomo_bp_kernel<<<std::min(tiles(31, 8 * kTomoBpRows, 1), 148u * 8), dim3(32, 8), 0, st>>>(
                d_img, d_sat, d_dc, d_src, d, b, c, tiled);
        }
    RN_CUDA_TRY(cudaGetLastError());
    return RN_OK;
}

static TomoDims tomo_dims(int nb, int nc, int nx, int ny, int nz, float dx, float dy, float dz, float cx, float cy,
                          float cz, int nu, int nview, int nv, float du, float dv, float off_u, float off_v) {
    TomoDims d;
    d.nb = nb; d.nc = nc; d.nx = nx; d.ny = ny; d.nz = nz;
    d.dx = dx; d.dy = dy; d.dz = dz; d.cx = cx; d.cy = cy; d.cz = cz;
    d.nu = nu; d.nview = nview; d.nv = nv;
    d.du = du; d.dv = dv; d.off_u = off_u; d.off_v = off_v;
    return d;
}

// Host-call scratch: grow-only device buffers guarded by a mutex.
struct TomoHost {
    std::mutex mu;
    cudaStream_t st = nullptr;
    void* buf[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    size_t cap[5] = {0, 0, 0, 0, 0};
    int ensure(int i, size_t bytes) {
        if (bytes <= cap[i]) return RN_OK;
        if (buf[i]) cudaFree(buf[i]);
        buf[i] = nullptr;
        cap[i] = 0;
        cudaError_t e = cudaMalloc(&buf[i], bytes);
        if (e != cudaSuccess) return set_cuda_error(e, "cudaMalloc");
        cap[i] = bytes;
        return RN_OK;
    }
};
static TomoHost g_tomo;

static int host_tomo(bool fp, float* out, const float* in, const float* dc, const float* sp, const TomoDims& d) {
    RN_TRY(tomo_validate(d));
    std::lock_guard<std::mutex> lk(g_tomo.mu);
    if (!g_tomo.st) RN_CUDA_TRY(cudaStreamCreateWithFlags(&g_tomo.st, cudaStreamNonBlocking));
    cudaStream_t st = g_tomo.st;
    size_t ni = (size_t)d.nb * d.nx * d.ny * d.nz * d.nc, np = (size_t)d.nb * d.nu * d.nview * d.nv * d.nc;
    size_t nsat = fp ? (size_t)d.nz * (d.nx + 1) * (d.ny + 1) : (size_t)d.nview * (d.nu + 1) * (d.nv + 1) + 2;
    RN_TRY(g_tomo.ensure(0, ni * 4));
    RN_TRY(g_tomo.ensure(1, np * 4));
    RN_TRY(g_tomo.ensure(2, (size_t)d.nview * 12));
    RN_TRY(g_tomo.ensure(3, (size_t)d.nview * 12));
    RN_TRY(g_tomo.ensure(4, nsat * 8));
    float* dimg = (float*)g_tomo.buf[0];
    float* dprj = (float*)g_tomo.buf[1];
    RN_CUDA_TRY(cudaMemcpyAsync(g_tomo.buf[2], dc, (size_t)d.nview * 12, cudaMemcpyHostToDevice, st));
    RN_CUDA_TRY(cudaMemcpyAsync(g_tomo.buf[3], sp, (size_t)d.nview * 12, cudaMemcpyHostToDevice, st));
    if (fp) {
        RN_CUDA_TRY(cudaMemcpyAsync(dimg, in, ni * 4, cudaMemcpyHostToDevice, st));
        RN_TRY(tomo_project(dprj, dimg, (float*)g_tomo.buf[2], (float*)g_tomo.buf[3], d, (double*)g_tomo.buf[4], st));
        RN_CUDA_TRY(cudaMemcpyAsync(out, dprj, np * 4, cudaMemcpyDeviceToHost, st));
    } else {
        RN_CUDA_TRY(cudaMemcpyAsync(dprj, in, np * 4, cudaMemcpyHostToDevice, st));
        RN_TRY(tomo_backproject(dimg, dprj, (float*)g_tomo.buf[2], (float*)g_tomo.buf[3], d, (double*)g_tomo.buf[4],
                                0, st));
        RN_CUDA_TRY(cudaMemcpyAsync(out, dimg, ni * 4, cudaMemcpyDeviceToHost, st));
    }
    RN_CUDA_TRY(cudaStreamSynchronize(st));
    return RN_OK;
}

}  // namespace rn

using namespace rn;

extern "C" {

int rn_tomo_sat_bytes(int nx, int ny, int nz, int nu, int nview, int nv, size_t* fp_bytes, size_t* bp_bytes) {
    if (fp_bytes) *fp_bytes = (size_t)nz * (nx + 1) * (ny + 1) * 8;
    if (bp_bytes) *bp_bytes = ((size_t)nview * (nu + 1) * (nv + 1) + 2) * 8;   // + 2 pad entries
    return RN_OK;
}

int rn_tomo_project(float* d_prj, const float* d_img, const float* d_detCenter, const float* d_src, double* d_sat,
                    int nBatches, int nChannels, int nx, int ny, int nz, float dx, float dy, float dz, float cx,
                    float cy, float cz, int nu, int nview, int nv, float du, float dv, float off_u, float off_v,
                    void* stream) {
    clear_error();
    if (!d_prj || !d_img || !d_detCenter || !d_src || !d_sat) return set_error(RN_ERR_ARG, "null argument");
    return tomo_project(d_prj, d_img, d_detCenter, d_src,
                        tomo_dims(nBatches, nChannels, nx, ny, nz, dx, dy, dz, cx, cy, cz, nu, nview, nv, du, dv,
                                  off_u, off_v),
                        d_sat, (cudaStream_t)stream);
}

int rn_tomo_backproject(float* d_img, const float* d_prj, const float* d_detCenter, const float* d_src, double* d_sat,
                        int nBatches, int nChannels, int nx, int ny, int nz, float dx, float dy, float dz, float cx,
                        float cy, float cz, int nu, int nview, int nv, float du, float dv, float off_u, float off_v,
                        int weightAllViews, void* stream) {
    clear_error();
    if (!d_prj || !d_img || !d_detCenter || !d_src || !d_sat) return set_error(RN_ERR_ARG, "null argument");
    return tomo_backproject(d_img, d_prj, d_detCenter, d_src,
                            tomo_dims(nBatches, nChannels, nx, ny, nz, dx, dy, dz, cx, cy, cz, nu, nview, nv, du, dv,
                                      off_u, off_v),
                            d_sat, weightAllViews ? 1 : 0, (cudaStream_t)stream);
}

void cDistanceDrivenTomoProjection(float* prj, const float* img, const float* detCenter, const float* src,
                                   int nBatches, int nChannels, int nx, int ny, int nz, float dx, float dy, float dz,
                                   float cx, float cy, float cz, int nu, int nview, int nv, float du, float dv,
                                   float off_u, float off_v) {
    clear_error();
    if (!prj || !img || !detCenter || !src) {
        set_error(RN_ERR_ARG, "null argument");
        return;
    }
    host_tomo(true, prj, img, detCenter, src,
              tomo_dims(nBatches, nChannels, nx, ny, nz, dx, dy, dz, cx, cy, cz, nu, nview, nv, du, dv, off_u, off_v));
}

void cDistanceDrivenTomoBackprojection(float* img, const float* prj, const float* detCenter, const float* src,
                                       int nBatches, int nChannels, int nx, int ny, int nz, float dx, float dy,
                                       float dz, float cx, float cy, float cz, int nu, int nview, int nv, float du,
                                       float dv, float off_u, float off_v) {
    clear_error();
    if (!prj || !img || !detCenter || !src) {
        set_error(RN_ERR_ARG, "null argument");
        return;
    }
    host_tomo(false, img, prj, detCenter, src,
              tomo_dims(nBatches, nChannels, nx, ny, nz, dx, dy, dz, cx, cy, cz, nu, nview, nv, du, dv, off_u, off_v));
}

}  // extern "C"
