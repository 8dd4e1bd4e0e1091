// Siddon cone-beam pair for upright detectors: every view's detector v axis
// runs along z and its u axis in the x-y plane (circular and other planar
// orbits).  All rays of a detector column iu then share one in-plane path, and
// along it ray iv rises linearly, so the in-plane tracing is done once per
// column and the rays (forward) or the voxels of one (x, y) (back) only follow
// their heights.
//
// Forward projection (cone_fp_col_kernel): a warp owns a detector column and
// 32 R of its rays, lanes along iv, the projections' contiguous axis.  It steps
// through the unit slabs along the in-plane axis on which this column advances
// most, so a slab crosses at most one grid line of the other axis; 32 slabs'
// image columns and crossing times are worked out at a time, one per lane, and
// broadcast from shared memory.  Voxels are read straight from the image: the
// lanes' voxels of one slab lie in one or two (x, y) columns, contiguous in z.
//
// Backprojection (cone_bp_col_kernel), the exact transpose as a gather.  On the
// part [t0, t1] of a slab that column iu spends above pixel (x, y), the rays
// below height q are those with iv < kappa(q, t), kappa(q, t) = (q - S_z) g(t)
// - c, g(t) = D_m / ((M + t) e_z).  With C(k) the prefix sums over iv of the
// rays' sinogram values times their lengths per slab,
//   F(q) = int_{t0}^{t1} C(kappa(q, t)) dt
// is the contribution below q, and voxel [q, q + 1] receives F(q + 1) - F(q).
// kappa hardly moves over the interval (by the rise of a ray inside one pixel),
// so F is (t1 - t0) C(k) plus, for the rare rays that cross height q over the
// pixel, the share of the interval they spend below it.  Lanes run along q;
// C and the sums over all views are FP64, and the differences are taken once at
// the end.  kappa is 64-bit fixed point (28 fractional bits), one wide integer
// multiply-add per face and interval end, good to 2.4e-7 rays and exact at the
// face level with the source: a level ray in that face belongs to the voxel
// above it, as in the forward projection.  The intervals
// of 32 views are worked out at a time, one view per lane.
//
// Measured, 256x256x128 voxels, 90 views of 512x128 cells: forward 1.77 ms
// (3.84 ms with one thread per ray stepping through global memory,
// cone_fp_kernel), back 3.52 ms with its table (19.8 ms with the shadow gather
// of cone_bp_kernel).  Both are bound by instruction issue and L1 reads.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "cone_internal.h"
#include "rn_device.cuh"
#include "rn_internal.h"

namespace rn {

constexpr int kColWarps = 8;

// In-plane path of detector column iu.
struct ColRay {
    double Dm, Da, ra;   // advance along the stepped axis, the other axis, and their ratio (|ra| <= 1)
    int m;               // the stepped axis
};
__device__ __forceinline__ ColRay col_ray(const ColView& V, int iu) {
    const double d0 = fma((double)iu, V.E[0], V.D[0]), d1 = fma((double)iu, V.E[1], V.D[1]);
    ColRay r;
    r.m = fabs(d0) >= fabs(d1) ? 0 : 1;
    r.Dm = r.m ? d1 : d0;
    r.Da = r.m ? d0 : d1;
    r.ra = r.Da / r.Dm;
    return r;
}

// `cnt` slabs of a warp's rays; kIn: no bounds checks on the heights.
template <int R, bool kIn>
__device__ __forceinline__ void col_slabs(float (&acc)[R], long long (&B)[R], const long long (&RB)[R],
                                          const float (&sb)[R], const float (&ob)[R], const float4* slabs, int cnt,
                                          const float* __restrict__ vol, int nc, int nz) {
    auto voxel = [&](int o, int b) {
        return kIn || (unsigned)b < (unsigned)nz ? __ldg(vol + (o + b * nc)) : 0.f;
    };
    for (int j = 0; j < cnt; j++) {
        const float4 e = slabs[j];
        const int o0 = __float_as_int(e.x), o1 = __float_as_int(e.y);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int b0 = (int)(B[r] >> 32);
            const float tb = fminf(fmaf(sb[r], __uint_as_float(0x3f800000u | ((unsigned)B[r] >> 9)), ob[r]), 1.f);
            B[r] += RB[r];
            const int b1 = (int)(B[r] >> 32);
            if (o1 == o0) {   // the same for the warp: one image column
                if (o0 >= 0) acc[r] = fmaf(tb, voxel(o0, b0), fmaf(1.f - tb, voxel(o0, b1), acc[r]));
            } else {
                const float t0 = fminf(e.z, tb), t1 = fmaxf(e.z, tb);
                const bool afirst = e.z < tb;
                const int om = afirst ? o1 : o0, bm = afirst ? b0 : b1;
                if (o0 >= 0) acc[r] = fmaf(t0, voxel(o0, b0), acc[r]);
                if (om >= 0) acc[r] = fmaf(t1 - t0, voxel(om, bm), acc[r]);
                if (o1 >= 0) acc[r] = fmaf(1.f - t1, voxel(o1, b1), acc[r]);
            }
        }
    }
}

template <int R>
__global__ void __launch_bounds__(32 * kColWarps) cone_fp_col_kernel(float* __restrict__ prj, const float* __restrict__ img,
                                                                      const ColView* __restrict__ views, ConeDims cd) {
    __shared__ float4 s_slab[kColWarps][32];   // voxel offsets of the two image columns (-1: outside) and the crossing time
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int iu = blockIdx.x * kColWarps + warp;
    if (iu >= cd.nu) return;   // the whole warp
    const int iv0 = blockIdx.y * 32 * R + lane;
    int zi = blockIdx.z;
    const int c = zi % cd.nc;
    zi /= cd.nc;
    const int view = zi % cd.nview, bt = zi / cd.nview;
    const ColView& V = views[view];
    const ColRay ray = col_ray(V, iu);
    const int m = ray.m;
    const double Sm = m ? V.S[1] : V.S[0], Sa = m ? V.S[0] : V.S[1], ra = ray.ra;
    const int nm = m ? cd.n[1] : cd.n[0], na = m ? cd.n[0] : cd.n[1], nz = cd.n[2];
    const int stm = (int)(m ? cd.st[1] : cd.st[0]), sta = (int)(m ? cd.st[0] : cd.st[1]);
    const float ira = fabs(ra) > 1e-30 ? (float)(1.0 / fabs(ra)) : 1e30f;
    // slabs whose part of the path can lie over the grid
    const double A0 = fma(-Sm, ra, Sa);   // lateral position at main coordinate 0
    int ks = 0, ke = nm;
    if (fabs(ra) > 1e-9) {
        const double k0 = -A0 / ra, k1 = (na - A0) / ra;
        ks = (int)fmin(fmax(floor(fmin(k0, k1)) - 1.0, 0.0), (double)nm);
        ke = (int)fmax(fmin(ceil(fmax(k0, k1)) + 1.0, (double)nm), 0.0);
    } else if (A0 < -1.0 || A0 > na + 1.0) {
        ke = 0;
    }
    // heights at the start of slab ks and their step per slab
    long long B[R], RB[R];
    float acc[R], irb[R], seg[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const double rz = fma((double)(iv0 + 32 * r), V.ez, V.dz0) / ray.Dm;
        B[r] = to_fixed(fma(ks - Sm, rz, V.Sz));
        RB[r] = to_fixed(rz);
        irb[r] = fabs(rz) > 1e-30 ? (float)(1.0 / fabs(rz)) : 1e30f;
        const double dm = m ? cd.d[1] : cd.d[0], da = m ? cd.d[0] : cd.d[1], dz = cd.d[2];
        seg[r] = (float)sqrt(dm * dm + ra * ra * da * da + rz * rz * dz * dz);
        acc[r] = 0.f;
    }
    // the time of the height crossing in a slab as one FMA on 1 + the position's
    // fraction; at or above 1 where there is none
    float sb[R], ob[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        sb[r] = RB[r] > 0 ? -irb[r] : irb[r];
        ob[r] = RB[r] > 0 ? 2.f * irb[r] : -irb[r];
    }
    const float* vol = img + bt * cd.img_b + c;
    const int nc = cd.nc;
    for (int kb = ks; kb < ke; kb += 32) {
        const int cnt = min(32, ke - kb);
        __syncwarp();
        if (lane < cnt) {
            const int k = kb + lane;
            const long long a0 = to_fixed(fma((double)k, ra, A0)), a1 = to_fixed(fma((double)(k + 1), ra, A0));
            const int c0 = (int)(a0 >> 32), c1 = (int)(a1 >> 32);
            const float fa = fixed_frac(a0);
            const float ta = c1 != c0 ? fminf((ra > 0 ? 1.f - fa : fa) * ira, 1.f) : 1.f;
            const int o0 = (unsigned)c0 < (unsigned)na ? c0 * sta + k * stm : -1;
            const int o1 = (unsigned)c1 < (unsigned)na ? c1 * sta + k * stm : -1;
            s_slab[warp][lane] = make_float4(__int_as_float(o0), __int_as_float(o1), ta, 0.f);
        }
        __syncwarp();
        // rays that stay inside the volume's height over these slabs need no bounds checks
        bool inside = true;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int b0 = (int)(B[r] >> 32), b1 = (int)((B[r] + cnt * RB[r]) >> 32);
            inside = inside && (unsigned)b0 < (unsigned)nz && (unsigned)b1 < (unsigned)nz;
        }
        if (__all_sync(0xffffffffu, inside))
            col_slabs<R, true>(acc, B, RB, sb, ob, s_slab[warp], cnt, vol, nc, nz);
        else
            col_slabs<R, false>(acc, B, RB, sb, ob, s_slab[warp], cnt, vol, nc, nz);
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int iv = iv0 + 32 * r;
        if (iv < cd.nv)
            prj[bt * cd.prj_b + (((long long)iu * cd.nview + view) * cd.nv + iv) * cd.nc + c] = acc[r] * seg[r];
    }
}

// C(k), k = 0 .. nv, of every (view, iu) for one (b, c): FP64 prefix sums over
// the rays in the order of increasing height of the sinogram value times the
// ray's length (mm) per slab of the view's main axis; *bad set where they are not
// finite.  One warp per (view, iu).
__global__ void __launch_bounds__(256) cone_col_table_kernel(double* __restrict__ tab, int* __restrict__ bad,
                                                             const float* __restrict__ prj,
                                                             const ColView* __restrict__ views, ConeDims cd, int bt,
                                                             int c) {
    const int lane = threadIdx.x & 31;
    const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= (long long)cd.nview * cd.nu) return;   // the whole warp
    const int view = (int)(row / cd.nu), iu = (int)(row - (long long)view * cd.nu);
    const ColView& V = views[view];
    const int m = V.m;
    const double Dm = fma((double)iu, m ? V.E[1] : V.E[0], m ? V.D[1] : V.D[0]);
    const double ra = fma((double)iu, m ? V.E[0] : V.E[1], m ? V.D[0] : V.D[1]) / Dm;
    const double dm = m ? cd.d[1] : cd.d[0], da = m ? cd.d[0] : cd.d[1], dz = cd.d[2];
    const double plane = dm * dm + ra * ra * da * da, idm = dz / Dm;
    const float* p = prj + bt * cd.prj_b + ((long long)iu * cd.nview + view) * cd.nv * cd.nc + c;
    double* t = tab + row * (cd.nv + 1);
    double carry = 0.0;
    if (lane == 0) t[0] = 0.0;
    for (int k0 = 0; k0 < cd.nv; k0 += 32) {
        const int k = k0 + lane;
        double w = 0.0;
        if (k < cd.nv) {
            const int iv = V.flip ? cd.nv - 1 - k : k;
            const double rise = fma((double)iv, V.ez, V.dz0) * idm;
            w = (double)__ldg(p + (long long)iv * cd.nc) * sqrt(fma(rise, rise, plane));
        }
        const double incl = carry + warp_incl_scan(w);
        if (k < cd.nv) t[k + 1] = incl;
        carry = __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0 && !isfinite(carry)) atomicOr(bad, 1);   // (one value of a sum is enough)
}

constexpr int kColFrac = 28;   // fractional bits of kappa

// One in-plane interval of a pixel: kappa at its two ends as a function of the
// face, kappa' = b + (q - z0) g in fixed point, raised by 2^28 - 1 so that its
// integer part counts the rays below the face; kappa + c at the first end and
// the difference of the two kappas as floats, a + (q - z0) ga and e + (q - z0) ge.
struct ColTask {
    longlong2 b;
    int4 g;        // g at the two ends, table row
    float4 f;      // a, ga, e, ge
    double t;      // length of the interval
};

// What face dq above z0 has below it: t C(k) into `sum` and t x the share of
// the rays that cross the face over the pixel into `part`.  kOne: at most one
// ray does (the heights that count move by less than one ray over a pixel).
template <bool kOne>
__device__ __forceinline__ void col_below(double& sum, float& part, const longlong2 b, const int4 g, const float4 f,
                                          double t, float tf, int dq, const double* __restrict__ tab, int nv) {
    const long long k0 = b.x + (long long)dq * g.x, k1 = b.y + (long long)dq * g.y;
    const int n0 = (int)(k0 >> kColFrac), n1 = (int)(k1 >> kColFrac);
    const float fq = (float)dq;
    // ray i crosses the face at the share s of the interval from its first
    // end: 1 / (kappa + c) is linear in t.  d0 = kappa_0 - i, d01 = kappa_0 -
    // kappa_1; kappa_0's fraction comes from its fixed point
    const float a0 = fmaf(fq, f.y, f.x), d01 = fmaf(fq, f.w, f.z);
    const float f1 = __uint_as_float(0x3f800000u | (((unsigned)k0 >> (kColFrac - 23)) & 0x7fffffu));   // 1 + fraction
    auto share = [&](float d0) {
        const float s = __saturatef(__fdividef(d0 * (a0 - d01), d01 * (a0 - d0)));
        return n0 > n1 ? s : 1.f - s;   // kappa falls: below until it crosses
    };
    const int lo = min(n0, n1);
    const double* row = tab + (long long)g.z * (nv + 1);
    if (kOne) {
        sum = fma(t, __ldg(row + min(max(lo, 0), nv)), sum);
        if (n0 != n1 && (unsigned)lo < (unsigned)nv)
            part = fmaf(tf * share(f1 - (n0 > n1 ? 1.f : 2.f)), (float)(__ldg(row + lo + 1) - __ldg(row + lo)), part);
    } else {
        const int l = min(max(lo, 0), nv), h = min(max(max(n0, n1), 0), nv);
        sum = fma(t, __ldg(row + l), sum);
        for (int i = l; i < h; i++)
            part = fmaf(tf * share((f1 - 1.f) + (float)(n0 - 1 - i)), (float)(__ldg(row + i + 1) - __ldg(row + i)), part);
    }
}

// One voxel by itself, from the projections: what the prefix sums cannot give where a
// value among them is not finite, since C(k) is then lost for every face above that
// ray.  Only the rays that meet the voxel count, each by its length in it.
__device__ double col_direct(const float* __restrict__ prj, const ColView* __restrict__ views,
                                          const ConeDims& cd, int x, int y, int z) {
    double acc = 0.0;
    for (int view = 0; view < cd.nview; view++) {
        const ColView& V = views[view];
        const int m = V.m;
        const double M = (m ? y : x) - V.S[m], A = V.S[1 - m] - (m ? x : y);
        double lo = 1e300, hi = -1e300;
        for (int k = 0; k < 4; k++) {   // as cone_bp_col_kernel finds the columns
            const double wm = M + (k & 1), wa = (k >> 1) - A;
            const double q = (V.D[1 - m] * wm - V.D[m] * wa) / (V.E[m] * wa - V.E[1 - m] * wm);
            lo = fmin(lo, q);
            hi = fmax(hi, q);
        }
        const int u0 = max(0, (int)ceil(fmax(lo - 2e-3, -1.0))), u1 = min(cd.nu - 1, (int)floor(fmin(hi + 2e-3, (double)cd.nu)));
        for (int iu = u0; iu <= u1; iu++) {
            const double Dm = fma((double)iu, V.E[m], V.D[m]), ra = fma((double)iu, V.E[1 - m], V.D[1 - m]) / Dm;
            const double xa = fma(ra, M, A);
            double ta = 0.0, tb = 1.0;
            if (fabs(ra) > 1e-12) {
                const double p = -xa / ra, q = (1.0 - xa) / ra;
                ta = fmax(0.0, fmin(p, q));
                tb = fmin(1.0, fmax(p, q));
            } else {
                const double xf = rint(xa * 4294967296.0);
                if (!(xf >= 0.0 && xf < 4294967296.0)) tb = -1.0;
            }
            if (!(tb - ta > 1e-12)) continue;
            // rays between the lowest and highest that reach the voxel over the pixel
            const double ga = Dm / ((M + ta) * V.ez), gb = Dm / ((M + tb) * V.ez), q0 = z - V.Sz, q1 = q0 + 1.0, c = V.dz0 / V.ez;
            const double vlo = fmin(fmin(q0 * ga, q1 * ga), fmin(q0 * gb, q1 * gb)) - c;
            const double vhi = fmax(fmax(q0 * ga, q1 * ga), fmax(q0 * gb, q1 * gb)) - c;
            const int v0 = max(0, (int)ceil(fmax(vlo - 1e-6, -1.0))), v1 = min(cd.nv - 1, (int)floor(fmin(vhi + 1e-6, (double)cd.nv)));
            const double dm = m ? cd.d[1] : cd.d[0], da = m ? cd.d[0] : cd.d[1], dz = cd.d[2];
            for (int iv = v0; iv <= v1; iv++) {
                const double rise = fma((double)iv, V.ez, V.dz0) / Dm, h = fma(rise, M, -q0);   // height over the voxel's face at t = 0
                double t0 = ta, t1 = tb;
                if (fabs(rise) > 1e-12) {
                    const double p = -h / rise, q = (1.0 - h) / rise;
                    t0 = fmax(t0, fmin(p, q));
                    t1 = fmin(t1, fmax(p, q));
                } else {
                    const double hf = rint(h * 4294967296.0);
                    if (!(hf >= 0.0 && hf < 4294967296.0)) continue;
                }
                if (t1 - t0 > 1e-9)
                    acc += (double)__ldg(prj + (((long long)iu * cd.nview + view) * cd.nv + iv) * cd.nc) * (t1 - t0) *
                           sqrt(dm * dm + ra * ra * da * da + rise * rise * dz * dz);
            }
        }
    }
    return acc;
}

// The slice whose projections hold a value that is not finite (*bad), a voxel per
// thread; cone_bp_col_kernel leaves it alone.
__global__ void __launch_bounds__(256) cone_bp_col_direct_kernel(float* __restrict__ img, const float* __restrict__ prj,
                                                                 const int* __restrict__ bad,
                                                                 const ColView* __restrict__ views, ConeDims cd, int bt,
                                                                 int c, int accumulate) {
    if (*bad == 0) return;
    const long long n = (long long)cd.n[0] * cd.n[1] * cd.n[2];
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
        const int z = (int)(i % cd.n[2]), y = (int)(i / cd.n[2] % cd.n[1]), x = (int)(i / cd.n[2] / cd.n[1]);
        const float v = (float)col_direct(prj + bt * cd.prj_b + c, views, cd, x, y, z);
        float* o = img + bt * cd.img_b + (long long)x * cd.st[0] + (long long)y * cd.st[1] + (long long)z * cd.nc + c;
        *o = accumulate ? *o + v : v;
    }
}

template <int R, bool kOne>
__global__ void __launch_bounds__(32 * kColWarps, 3) cone_bp_col_kernel(float* __restrict__ img, const double* __restrict__ tab,
                                                                      const int* __restrict__ bad,
                                                                      const ColView* __restrict__ views, ConeDims cd,
                                                                      int bt, int c, int accumulate) {
    __shared__ ColTask s_task[kColWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // 4 x 2 neighbouring pixels per block: they read neighbouring rows of the table
    const int x = blockIdx.x * 4 + (warp & 3), y = blockIdx.y * 2 + (warp >> 2);
    if (x >= cd.n[0] || y >= cd.n[1] || *bad) return;   // the whole warp
    const int nz = cd.n[2], z0 = blockIdx.z * 32 * R;
    const int top = min(nz - z0, 32 * R);   // the chunk's upper face, evaluated by the lanes' own views
    double acc[R], acct = 0.0;
    float part[R], partt = 0.f;
#pragma unroll
    for (int r = 0; r < R; r++) {
        acc[r] = 0.0;
        part[r] = 0.f;
    }
    ColTask* task = s_task[warp];
    for (int vb = 0; vb < cd.nview; vb += 32) {
        const int view = vb + lane;
        // detector columns whose rays can meet the pixel: its corners seen from the source
        int u0 = 1, u1 = 0;
        double Dm0 = 0, Em = 0, Da0 = 0, Ea = 0, M = 0, A = 0, iez = 0, zr = 0, cc = 0;
        int zb = 0;   // the face of this chunk next to the source's height
        if (view < cd.nview) {
            const ColView& V = views[view];
            const int m = V.m;
            Dm0 = V.D[m];
            Em = V.E[m];
            Da0 = V.D[1 - m];
            Ea = V.E[1 - m];
            M = (m ? y : x) - V.S[m];
            A = V.S[1 - m] - (m ? x : y);
            iez = V.iez;
            // kappa is worked out from the face at the source's height, where a level
            // ray lies exactly in the face and no rounding may push it below
            zb = (int)fmin(fmax(rint(V.Sz) - z0, 0.0), 32.0 * R);
            zr = (z0 + zb) - V.Sz;
            cc = V.c;
            float lo = 1e30f, hi = -1e30f;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                // iu of the in-plane ray through (M + k0, k1 - A) from the source
                const double wm = M + (k & 1), wa = (k >> 1) - A;
                const float q = __fdividef((float)(Da0 * wm - Dm0 * wa), (float)(Em * wa - Ea * wm));
                lo = fminf(lo, q);
                hi = fmaxf(hi, q);
            }
            u0 = max(0, (int)ceilf(fmaxf(lo - 2e-3f, -1.f)));
            u1 = min(cd.nu - 1, (int)floorf(fminf(hi + 2e-3f, (float)cd.nu)));
        }
        for (int iu = u0;; iu++) {
            if (!__any_sync(0xffffffffu, iu <= u1)) break;
            bool hit = false;
            ColTask T;
            if (iu <= u1) {
                const double Dm = fma((double)iu, Em, Dm0), Da = fma((double)iu, Ea, Da0);
                const double ra = Da / Dm, xa = fma(ra, M, A);   // lateral offset at the pixel's low face
                double ta = 0.0, tb = 1.0;
                if (fabs(ra) > 1e-12) {
                    const double ir = 1.0 / ra, p = -xa * ir, q = (1.0 - xa) * ir;
                    ta = fmax(0.0, fmin(p, q));
                    tb = fmin(1.0, fmax(p, q));
                } else {
                    // along the other axis's grid lines: in or beside the pixel by the
                    // position as the forward projection rounds it
                    const double xf = rint(xa * 4294967296.0);
                    if (!(xf >= 0.0 && xf < 4294967296.0)) tb = -1.0;
                }
                hit = tb - ta > 1e-12;
                if (hit) {
                    const double s = Dm * iez, g0 = s / (M + ta), g1 = s / (M + tb);
                    constexpr double kOneFixed = (double)(1 << kColFrac);
                    const int i0 = (int)llrint(g0 * kOneFixed), i1 = (int)llrint(g1 * kOneFixed);
                    T.b = make_longlong2(llrint((zr * g0 - cc) * kOneFixed) + ((1 << kColFrac) - 1) - (long long)zb * i0,
                                         llrint((zr * g1 - cc) * kOneFixed) + ((1 << kColFrac) - 1) - (long long)zb * i1);
                    T.g = make_int4(i0, i1, view * cd.nu + iu, 0);
                    const double za = zr - zb;
                    T.f = make_float4((float)(za * g0), (float)g0, (float)(za * (g0 - g1)), (float)(g0 - g1));
                    T.t = tb - ta;
                    col_below<kOne>(acct, partt, T.b, T.g, T.f, T.t, (float)T.t, top, tab, cd.nv);
                }
            }
            const unsigned hits = __ballot_sync(0xffffffffu, hit);
            __syncwarp();   // the previous round's tasks have been read
            if (hit) task[__popc(hits & ((1u << lane) - 1))] = T;
            __syncwarp();
            const int n = __popc(hits);
            for (int e = 0; e < n; e++) {
                const longlong2 b = task[e].b;
                const int4 g = task[e].g;
                const float4 f = task[e].f;
                const double t = task[e].t;
                const float tf = (float)t;
#pragma unroll
                for (int r = 0; r < R; r++)
                    col_below<kOne>(acc[r], part[r], b, g, f, t, tf, lane + 32 * r, tab, cd.nv);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        acct += __shfl_xor_sync(0xffffffffu, acct, o);
        partt += __shfl_xor_sync(0xffffffffu, partt, o);
    }
    float* out = img + bt * cd.img_b + (long long)x * cd.st[0] + (long long)y * cd.st[1] + c;
#pragma unroll
    for (int r = 0; r < R; r++) {
        // the voxel's upper face: the next lane's, the next 32 faces' first, or the chunk's top
        const int rn = r + 1 < R ? r + 1 : r;
        const double up = __shfl_down_sync(0xffffffffu, acc[r], 1), over = __shfl_sync(0xffffffffu, acc[rn], 0);
        const float upp = __shfl_down_sync(0xffffffffu, part[r], 1), overp = __shfl_sync(0xffffffffu, part[rn], 0);
        const int dz = lane + 32 * r;
        if (dz < top) {
            const bool last = dz + 1 == top;
            const double hi = last ? acct : lane == 31 ? over : up;
            const float hip = last ? partt : lane == 31 ? overp : upp;
            float* o = out + (long long)(z0 + dz) * cd.nc;
            const float v = (float)(hi - acc[r]) + (hip - part[r]);
            *o = accumulate ? *o + v : v;
        }
    }
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
// The limits: the detector's v exactly along z and its u exactly in the plane;
// every in-plane path that meets the grid crosses it between the source and
// the detector; rays rise by at most one voxel per in-plane voxel step; and
// kappa fits its fixed point (under 7.9 rays per voxel height, and under 3.9
// rays crossed inside one pixel).  Anything else stays on the general kernels.
bool cone_col_views(const std::vector<ConeView>& views, const ConeDims& cd, std::vector<ColView>& out, bool& one) {
    out.clear();
    one = true;
    const double nx = cd.n[0], ny = cd.n[1], nz = cd.n[2];
    if ((long long)cd.nview * cd.nu > 0x7fffffff || (long long)cd.nview * cd.nb * cd.nc > 65535) return false;
    if (cd.n[1] > 2 * 65535 || cd.n[2] > 32 * 65535) return false;   // the grid's y and z
    for (const ConeView& v : views) {
        if (v.m == 2 || v.Ev[0] != 0.0 || v.Ev[1] != 0.0 || v.Eu[2] != 0.0 || v.Ev[2] == 0.0) return false;
        ColView q;
        for (int k = 0; k < 2; k++) {
            q.S[k] = v.S[k];
            q.D[k] = v.C[k] - v.S[k];
            q.E[k] = v.Eu[k];
        }
        q.Sz = v.S[2];
        q.dz0 = v.C[2] - v.S[2];
        q.ez = v.Ev[2];
        q.flip = q.ez < 0;
        const double ez = std::fabs(q.ez), first = q.flip ? q.dz0 + (cd.nv - 1) * q.ez : q.dz0;
        q.c = first / ez;
        q.iez = 1.0 / ez;
        q.m = v.m;
        const double rise = std::max(std::fabs(q.dz0), std::fabs(q.dz0 + (cd.nv - 1) * q.ez));
        for (int iu = 0; iu < cd.nu; iu++) {
            const double D[2] = {q.D[0] + iu * q.E[0], q.D[1] + iu * q.E[1]};
            if (!(rise <= std::max(std::fabs(D[0]), std::fabs(D[1])))) return false;
            // the infinite line's passage over the grid, as parameters of the segment
            double t0 = -1e300, t1 = 1e300;
            const double n[2] = {nx, ny};
            for (int k = 0; k < 2; k++) {
                if (D[k] == 0.0) {
                    if (q.S[k] < 0 || q.S[k] > n[k]) t1 = -1e300;
                    continue;
                }
                const double a = -q.S[k] / D[k], b = (n[k] - q.S[k]) / D[k];
                t0 = std::max(t0, std::min(a, b));
                t1 = std::min(t1, std::max(a, b));
            }
            if (t1 > t0 && !(t0 > 0.0 && t1 < 1.0)) return false;
        }
        // the grid on one side of the line through the source along u, so that
        // every pixel corner has its detector column
        double side[4];
        for (int k = 0; k < 4; k++)
            side[k] = q.E[0] * ((k >> 1) * (ny + 2) - 1 - q.S[1]) - q.E[1] * ((k & 1) * (nx + 2) - 1 - q.S[0]);
        if (!(*std::min_element(side, side + 4) > 0.0 || *std::max_element(side, side + 4) < 0.0)) return false;
        // distance shares (M + t) / D_m over the grid
        double lmin = 1e300, mmin = 1e300;
        const int m = v.m;
        for (int iu : {0, cd.nu - 1})
            for (double pm : {0.0, (double)cd.n[m]}) {
                const double M = pm - q.S[m], Dm = q.D[m] + iu * q.E[m];
                lmin = std::min(lmin, M / Dm);
                mmin = std::min(mmin, std::fabs(M));
            }
        if (!(lmin > 0.0)) return false;
        const double g = 1.0 / (lmin * ez), zmax = std::max(std::fabs(q.Sz), std::fabs(nz + 128 - q.Sz));
        if (!(g < 7.9 && mmin > 1.0 && zmax * g / mmin < 3.9 && zmax * g < 1e6 && std::fabs(q.c) < 1e6)) return false;
        one = one && std::max(std::fabs(q.Sz), std::fabs(nz - q.Sz)) * g / mmin < 0.99;
        out.push_back(q);
    }
    return true;
}

int cone_col_project(const ColView* d_views, const ConeDims& cd, float* d_prj, const float* d_img, cudaStream_t st) {
    // two rays per lane where the detector has more than 32 rows
    const unsigned gx = (unsigned)((cd.nu + kColWarps - 1) / kColWarps), gz = (unsigned)(cd.nview * cd.nb * cd.nc);
    if (cd.nv > 32)
        cone_fp_col_kernel<2><<<dim3(gx, (unsigned)((cd.nv + 63) / 64), gz), 32 * kColWarps, 0, st>>>(d_prj, d_img,
                                                                                                       d_views, cd);
    else
        cone_fp_col_kernel<1><<<dim3(gx, 1, gz), 32 * kColWarps, 0, st>>>(d_prj, d_img, d_views, cd);
    RN_CUDA_TRY(cudaGetLastError());
    return RN_OK;
}

static size_t col_table_entries(const ConeDims& cd) { return (size_t)cd.nview * cd.nu * (cd.nv + 1); }
size_t cone_col_table_bytes(const ConeDims& cd) { return sizeof(double) * (col_table_entries(cd) + 1); }   // and the flag

template <int R>
static void launch_bp_col(const dim3& grid, const ColView* d_views, const ConeDims& cd, bool one, const double* d_tab,
                          const int* d_bad, float* d_img, int accumulate, int b, int c, cudaStream_t st) {
    if (one)
        cone_bp_col_kernel<R, true><<<grid, 32 * kColWarps, 0, st>>>(d_img, d_tab, d_bad, d_views, cd, b, c, accumulate);
    else
        cone_bp_col_kernel<R, false><<<grid, 32 * kColWarps, 0, st>>>(d_img, d_tab, d_bad, d_views, cd, b, c, accumulate);
}

int cone_col_backproject(const ColView* d_views, const ConeDims& cd, bool one, double* d_tab, float* d_img,
                         const float* d_prj, int accumulate, cudaStream_t st) {
    const long long rows = (long long)cd.nview * cd.nu;
    int* d_bad = reinterpret_cast<int*>(d_tab + col_table_entries(cd));
    const int R = cd.n[2] > 64 ? 4 : cd.n[2] > 32 ? 2 : 1;
    const dim3 grid((unsigned)((cd.n[0] + 3) / 4), (unsigned)((cd.n[1] + 1) / 2),
                    (unsigned)((cd.n[2] + 32 * R - 1) / (32 * R)));
    for (int b = 0; b < cd.nb; b++)
        for (int c = 0; c < cd.nc; c++) {
            RN_CUDA_TRY(cudaMemsetAsync(d_bad, 0, sizeof(int), st));
            cone_col_table_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(d_tab, d_bad, d_prj, d_views, cd, b, c);
            if (R == 4) launch_bp_col<4>(grid, d_views, cd, one, d_tab, d_bad, d_img, accumulate, b, c, st);
            else if (R == 2) launch_bp_col<2>(grid, d_views, cd, one, d_tab, d_bad, d_img, accumulate, b, c, st);
            else launch_bp_col<1>(grid, d_views, cd, one, d_tab, d_bad, d_img, accumulate, b, c, st);
            cone_bp_col_direct_kernel<<<148 * 8, 256, 0, st>>>(d_img, d_prj, d_bad, d_views, cd, b, c, accumulate);
        }
    RN_CUDA_TRY(cudaGetLastError());
    return RN_OK;
}

}  // namespace rn
