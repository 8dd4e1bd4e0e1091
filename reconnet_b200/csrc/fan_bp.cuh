// Per-view device code shared by the fan backprojection kernels (fan.cu,
// fan_group.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "rn_device.cuh"
#include "rn_internal.h"

namespace rn {

// Per-view parameters the BP inner loop reads, staged in shared memory.
struct BpView {
    double pard, perpd;   // source coordinates (Siddon band positions)
    float par, perp, kappa, tA, tB, sigma, round;
    int xcls;
    int good;             // the polynomial is good over the whole tile
    int inside;           // the window holds every entry that the tile's edge-index cubics can select
};

// V views per staged chunk.
template <int V>
struct BpSharedT {
    ViewGeo rec[2][V];   // view records staged for the next chunk
    uint64_t bars[2];
    int elo[3][V];       // first staged table entry per view
    BpView vw[3][V];
};

// Edge index t of the matched parametrisation for a slope r
// (r = (q - par) / (l - perp) at lattice point (line l, position q)).
__device__ __forceinline__ float matched_t(const ViewGeo& vg, float r) {
    return vg.tA + vg.tB * atanf(vg.kappa * r);
}

// Edge index t(r) = tA + tB atan(kappa r) as a cubic around the slope r_t at
// the lane's middle lattice point: along one lane the lattice points differ
// in one coordinate only.  It is off by at most 4.7 / 24 |tB| h^4 cells for slopes h
// / kappa from the middle: 4e-5 over 17 points of a 512 x 512 image of 0.7 mm pixels
// 595 mm from the source, but a cell and more where the image comes close to it.  The
// Siddon and pixel-driven kernels, and the matched one for points 4 from the middle,
// only select a cell with it and are exact inside; reference mode (fan.cu,
// fan_group.cu) takes an interval's ends from it, where the shift cancels between the
// two but for its change over a pixel.
struct TCubic {
    float rt, c0, c1, c2, c3;
};
__device__ __forceinline__ TCubic t_cubic(const BpView& vg, float rt) {
    const float ut = vg.kappa * rt;
    const float iw = __fdividef(1.0f, fmaf(ut, ut, 1.0f));
    const float k1 = vg.tB * vg.kappa * iw;
    TCubic c;
    c.rt = rt;
    c.c0 = fmaf(vg.tB, atanf(ut), vg.tA);
    c.c1 = k1;
    c.c2 = -k1 * vg.kappa * ut * iw;
    c.c3 = k1 * vg.kappa * vg.kappa * (fmaf(3.0f * ut, ut, -1.0f) * (1.0f / 3.0f)) * iw * iw;
    return c;
}

// floor(x) for |x| < 2^22 on the FMA / ALU pipes (round-down add of 1.5 * 2^23).
__device__ __forceinline__ int floor_small(float x) {
    return __float_as_int(__fadd_rd(x, 12582912.0f)) - 0x4B400000;
}

__device__ __forceinline__ void split_hilo(double v, float& h, float& l) {
    h = (float)v;
    l = (float)(v - (double)h);
}

// s + e = a + b exactly (TwoSum).
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// Warp 0 of a backprojection CTA prepares chunk c (views c * V ...) of its tile
// of kCols x kRows pixels at (X0, Y0): lane = view * 4 + tile corner evaluates
// the edge index at its corner, a 4-lane min gives the first staged table entry
// (edge 0 is entry `pad`; `back` entries of slack before it), and the
// view's parameters go to slot c % 3.  kPoly 3 or 4: also whether the window holds
// every entry that a cubic (quartic) index of the tile can select.  Kept out of
// line: it runs once per chunk in one warp, and inlined its temporaries would raise the
// register count of the whole accumulation loop.
template <int V, int kCols, int kRows, int kPoly = 0>
__device__ __noinline__ void bp_prep(BpSharedT<V>* sh, const ViewGeo* src, int c, int nview, int X0, int Y0,
                                     int nx, int ny, int tabn, int win, int pad, int back) {
    const int lane = threadIdx.x & 31, v = lane >> 2, corner = lane & 3;
    const bool valid = v < V && c * V + v < nview;
    const ViewGeo& vg = src[valid ? v : 0];
    const int cx = corner & 1, cy = corner >> 1;
    const int xcls = vg.xcls;
    // the tile's corners; cut to the image unless the polynomial (and with it an
    // unclamped index of a lane beyond the image) is good over the whole tile,
    // which may reach past the source
    const bool whole = kPoly && (kPoly == 4 ? vg.quartic : vg.cubic);
    const float X = (float)(whole ? X0 + cx * kCols : min(X0 + cx * kCols, nx));
    const float Y = (float)(whole ? Y0 + cy * kRows : min(Y0 + cy * kRows, ny));
    const float l = xcls ? Y : X, q = xcls ? X : Y;
    float t = matched_t(vg, (q - (float)vg.par) / (l - (float)vg.perp));
    float tmax = t;
    if (kPoly) {
        tmax = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, 1));
        tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 2));
    }
    t = fminf(t, __shfl_xor_sync(0xffffffffu, t, 1));
    t = fminf(t, __shfl_xor_sync(0xffffffffu, t, 2));
    if (valid && corner == 0) {
        const int slot = c % 3;
        const int lo = (int)floorf(t) + pad - back;
        sh->elo[slot][v] = max(0, min(lo, tabn - win));
        BpView& w = sh->vw[slot][v];
        // (an index may be a quarter of a cell off, hence one entry of room each side)
        if (kPoly) w.good = whole;
        if (kPoly)
            w.inside = whole && back >= 1 && lo >= 0 && lo < tabn - win && tmax < 1e6f &&
                       (int)floorf(tmax) + pad + 1 < lo + win;
        w.pard = vg.par;
        w.perpd = vg.perp;
        w.par = (float)vg.par;
        w.perp = (float)vg.perp;
        w.kappa = vg.kappa;
        w.tA = vg.tA;
        w.tB = vg.tB;
        w.sigma = vg.sigma;
        w.round = vg.round;
        w.xcls = vg.xcls;
    }
}

}  // namespace rn
