// What the Siddon cone-beam kernels share: per-view geometry, dimensions and
// the fixed-point positions along a ray.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "rn_internal.h"

namespace rn {

struct ConeView {
    double S[3];              // source, voxel coordinates
    double C[3];              // end point of ray (iu, iv) = (0, 0), voxel coordinates
    double Eu[3], Ev[3];      // end-point step per detector index along u / v
    float Sh[3], Sl[3];       // source as hi / lo floats
    float au[4], av[4], ad[4];   // shadow: iu = (au . P + au[3]) / (ad . P + ad[3]), iv likewise
    float ulo, uhi, vlo, vhi, dlo, dhi;   // sums of min(0, a_k) / max(0, a_k) over the three axes
    // separable views (affine = 1 or 2): every ray advances by the same Dm0
    // along m, and r_a = rho[0] + iu rho[1] + iv rho[2], r_b = rho[3] +
    // iu rho[4] + iv rho[5] with rho[2] = rho[4] = 0 (affine = 1: a follows
    // iu, b follows iv) or rho[1] = rho[5] = 0 (affine = 2)
    double rho[6];
    double Dm0;
    int m, a, b, affine;
};

struct ConeDims {
    int n[3];
    float d[3];
    long long st[3];          // image strides (elements) along x, y, z
    int nc, nu, nv, nview, nb;
    long long img_b, prj_b;   // batch strides
};

__device__ __forceinline__ long long to_fixed(double v) { return llrint(v * 4294967296.0); }

// Fractional part of a fixed-point position as a float in [0, 1) (its top 23
// bits: exact to 1.2e-7).
__device__ __forceinline__ float fixed_frac(long long p) {
    return __uint_as_float(0x3f800000u | ((unsigned)p >> 9)) - 1.0f;
}

// ---------------------------------------------------------------------------
// Upright detectors (cone_col.cu): every view's v axis along z, its u axis and
// main axis in the x-y plane, so the in-plane path of a ray depends on iu only.
// ---------------------------------------------------------------------------
struct ColView {
    double S[2], D[2], E[2];   // in-plane source, C - S and the step per iu, voxels
    double Sz;                 // source height, voxels
    double dz0, ez;            // height of ray iv's end point over the source: dz0 + iv ez (voxels)
    double c, iez;             // the same with ez > 0 (rays renumbered where flip): dz0' / ez', 1 / ez'
    int m, flip;
};
// Fills `out` where the column kernels can take the plan (false otherwise);
// `one`: no height moves over more than one ray inside a pixel.
bool cone_col_views(const std::vector<ConeView>& views, const ConeDims& cd, std::vector<ColView>& out, bool& one);
int cone_col_project(const ColView* d_views, const ConeDims& cd, float* d_prj, const float* d_img, cudaStream_t st);
size_t cone_col_table_bytes(const ConeDims& cd);
int cone_col_backproject(const ColView* d_views, const ConeDims& cd, bool one, double* d_tab, float* d_img,
                         const float* d_prj, int accumulate, cudaStream_t st);

// ---------------------------------------------------------------------------
// Tomosynthesis (cone_tile.cu): z the main axis, u along x, v along y.
// ---------------------------------------------------------------------------
struct TileView {
    double su, sv, sm;             // source, voxels (x, y, z)
    double ru0, ru1, rv0, rv1;     // slopes ru0 + iu ru1 along x and rv0 + iv rv1 along y, per slab
    float gu_max, gv_max;          // widest ray spacing inside the grid, voxels
    int vt;                        // the row whose rays are (the closest to) level along y
};
struct TilePlan {
    bool fp_narrow = false;        // rays under a voxel apart
    double gu = 1, gv = 1;         // widest ray spacing, voxels
    int kv = 0;                    // rows of rays that can meet one voxel
    int bp_patch = 0, bp_smem = 0; // floats of a backprojection patch, shared memory of a block
};
// Fills `out` and `tp` where the tile kernels can take the plan (false otherwise).
bool cone_tile_views(const std::vector<ConeView>& views, const ConeDims& cd, std::vector<TileView>& out, TilePlan& tp);
// whether the forward projection goes in tiles of 64 x 128 rays (else 32 x 64)
bool cone_tile_big(const ConeDims& cd, const TilePlan& tp);
int cone_tile_attributes();
size_t cone_tile_fp_bytes(const ConeDims& cd);
size_t cone_tile_bp_bytes(const ConeDims& cd);
int cone_tile_project(const TileView* d_views, const ConeDims& cd, const TilePlan& tp, float* d_vol, float* d_prj,
                      const float* d_img, cudaStream_t st);
int cone_tile_backproject(const TileView* d_views, const ConeDims& cd, const TilePlan& tp, float* d_wp, float* d_img,
                          const float* d_prj, int accumulate, cudaStream_t st);

}  // namespace rn
