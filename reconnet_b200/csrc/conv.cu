// BF16 3x3 convolutions of the learned prior on the 5th-generation tensor
// cores (tcgen05.mma, FP32 accumulators in tensor memory), with the input
// tiles brought in by TMA tensor copies from this GPU's own memory.
//
// The prior is a small residual CNN (5 layers of 3x3 convolutions, 32
// channels, ReLU; in 1 channel, out 1 channel plus the input).  It has no
// counterpart among the reference's kernels: the reference's learned use of
// the projectors goes through TensorFlow (python/ReconNet.py:773-830, the
// projector pair as differentiable ops) and its prior solvers are dictionary
// and low-rank methods (PriorFunctionSolver/omp.cu, NuclearNormSoftThresh.cu).
//
// Activation layout ("blocked"): bf16 [N][C/8][H][W][8] -- 16 bytes per pixel
// and channel chunk.  A TMA box of 3 image rows x (128 + 2) pixels x C/8
// chunks lands in shared memory as [chunk][row][pixel][8 channels]: 16-byte
// runs of 8 channels, consecutive pixels 16 bytes apart.  That is a canonical
// no-swizzle operand layout for the tensor core as it stands:
//   forward / input gradient, D[pixel][co] = sum_k A[pixel][k] B[co][k], A
//   K-major: for tap (dy, dx) and chunk c the 128 pixels of the tile are 128
//   consecutive 16-byte rows starting at pixel dx of row dy -- the im2col
//   matrix is read in place, with no copy;
//   weight gradient, D[co][(tap, ci)] = sum_p dY[p][co] X[p + tap][ci], both
//   operands MN-major: 8 pixels x 8 channels per 128-byte core matrix.
// Zero padding at the image border is the TMA's out-of-bounds fill.
//
// Descriptor bit layouts (instruction descriptor of kind::f16, shared-memory
// matrix descriptor version 1 for sm_100) follow the PTX ISA for tcgen05.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <string>

#include "rn_device.cuh"
#include "rn_internal.h"

namespace rn {

constexpr int kConvThreads = 128;     // one warpgroup: the 128 accumulator lanes
constexpr int kConvTile = 128;        // output pixels per tile (MMA M)
constexpr int kBoxW = kConvTile + 2;  // pixels per box row (halo of one on each side)
constexpr int kWgStages = 4;          // stages of the weight gradient's load pipeline
constexpr int kZeroBytes = 2048;      // zero rows standing in for the tenth tap of an 8-channel layer

// ---- tcgen05 / TMA primitives ------------------------------------------------
// (addresses and offsets stay below 2^18 bytes, so sums of low words do not carry
// between their fields)
__host__ __device__ constexpr uint32_t desc_lo(uint32_t offset, uint32_t lbo) { return (offset >> 4) + ((lbo >> 4) << 16); }
__host__ __device__ constexpr uint32_t desc_hi(uint32_t sbo) { return (sbo >> 4) | (1u << 14); }   // version 1, no swizzle

// one lane of the (converged) warp
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}

// kind::f16 instruction descriptor: BF16 A and B, FP32 D, M = 128.
__host__ __device__ constexpr uint32_t umma_idesc(int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// Matrix descriptors are given as their low word (start address and leading
// byte offset: the loops add constants to it) and their constant high word.
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint32_t da_lo, uint32_t da_hi, uint32_t db_lo,
                                          uint32_t db_hi, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "mov.b64 a, {%1, %2};\n\t"
        "mov.b64 b, {%3, %4};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}" ::"r"(tmem_d),
        "r"(da_lo), "r"(da_hi), "r"(db_lo), "r"(db_hi), "r"(idesc), "r"(accum));
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 32 lanes x 32 consecutive FP32 columns: thread t of the warp gets lane (base lane + t).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, "
        "%6}], [%7];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ uint4 pack_bf16x8(const float* v) {
    uint4 o;
    uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    return o;
}
__device__ __forceinline__ void unpack_bf16x8(uint4 u, float* v) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&w[i]);
        float2 f = __bfloat1622float2(h);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}

// Offset (bytes) in a box [CH][3][boxw][16 B] of tap t's first chunk for
// output pixel 0; tap 9 (the padding of an 8-channel layer) is the zero rows.
__device__ __forceinline__ uint32_t tap_off(int t, int ch, int boxw = kBoxW) {
    if (t >= 9) return (uint32_t)(ch * 3 * boxw * 16);
    return (uint32_t)(((t / 3) * boxw + (t % 3)) * 16);
}

// The tiles of a CTA, blockIdx.x + i gridDim.x over (n, h, tw) with tw fastest:
// the coordinates step by the grid's own, with carries.  (Dividing a 64-bit
// tile index out for every tile cost the producer and the epilogue about a
// thousand cycles of latency each per tile.)
struct TileWalk {
    int tw, h, n;
    int stw, sh, sn, tiles_w, H;
    __device__ __forceinline__ TileWalk(long long first, long long step, int tiles_w_, int H_) : tiles_w(tiles_w_), H(H_) {
        tw = (int)(first % tiles_w);
        h = (int)(first / tiles_w % H);
        n = (int)(first / tiles_w / H);
        stw = (int)(step % tiles_w);
        sh = (int)(step / tiles_w % H);
        sn = (int)(step / tiles_w / H);
    }
    __device__ __forceinline__ void next() {
        tw += stw;
        h += sh;
        n += sn;
        if (tw >= tiles_w) {
            tw -= tiles_w;
            h++;
        }
        if (h >= H) {
            h -= H;
            n++;
        }
    }
};

// ---- forward / input-gradient convolution --------------------------------------
// mode 0: out bf16 blocked = relu(conv + bias); mode 1: out fp32 [N][H][W] =
// conv[0] + bias[0] + aux (the residual); mode 2: out bf16 blocked = conv *
// (aux > 0), aux the bf16 blocked activation (ReLU mask of the input
// gradient); mode 3: out fp32 [N][cout][H][W] = conv + bias (tests).
struct ConvArgs {
    void* out;
    const uint4* wpack;   // B operand image: [kchunks][NPAD][16 B]
    const float* bias;    // [cout] or null
    const void* aux;
    int N, H, W;
    int cout;             // real output channels (1 or multiple of 8)
    int mode;
    int* err;
};

// Warp-specialised pipeline.  Warp 9 loads: it keeps kConvStages TMA boxes in
// flight, refilling a stage when its "empty" barrier says that the MMAs on it are
// done.  Warp 8 issues each tile's MMA group (one elected lane) and commits it
// twice, to the box's "empty" barrier and to the accumulator's "full" barrier.
// Warps 0-3 and 4-7 are the epilogues of the even and the odd tiles: thread t
// reads TMEM lane t (output pixel w0 + t of the tile's row) from its accumulator
// of 32 columns, releases the accumulator (one arrival per warp on its "empty"
// barrier) and stores.  So
// the TMA copies, the MMAs of tile i and the epilogue of tile i - 1 overlap.
// What bounded it were serial instruction streams: a lane that loaded and issued
// from 64-bit indices, then one warpgroup's epilogues.  8 images of 512 x 512, 32
// to 32 channels: 128 us with both, 82 us with loads in their own warp and
// descriptors as a base and constants, 66 us with a warpgroup per accumulator; a
// tile's 18 MMAs read 128 x 16 operands from shared memory for 720 of its 1130
// cycles on the SM.
//
// Boxes: the tensor map views each image row as groups of PIX pixels (16 PIX
// bytes; PIX = 8 when the width allows, else 2, else 1), so a TMA row is a
// whole 128-byte line rather than half a 32-byte sector.  A box then starts
// PIX - 1 pixels before the halo pixel w0 - 1 (128 + 2 PIX pixels) and the
// operands start 16 (PIX - 1) bytes into each box row.
constexpr int kConvStages = 3;
constexpr int kConvEpilogues = 2;   // epilogue warpgroups, one per accumulator
constexpr int kConvWsThreads = kConvEpilogues * kConvThreads + 64;

template <int CH, int NPAD, int PIX>
__global__ void __launch_bounds__(kConvWsThreads) conv3x3_kernel(const __grid_constant__ CUtensorMap tm_in, ConvArgs a) {
    constexpr int KSTEPS = CH == 4 ? 18 : 5;
    constexpr int KCH = 2 * KSTEPS;                              // B chunks (the last one of an 8-channel layer is zero)
    constexpr int BOXW = kConvTile + 2 * PIX;                    // pixels per box row
    constexpr uint32_t A0 = 16 * (PIX - 1);                      // the operands' first pixel within a box row
    constexpr uint32_t BOX_BYTES = CH * 3 * BOXW * 16;
    constexpr uint32_t BOX_ALLOC = (BOX_BYTES + kZeroBytes + 1023) & ~1023u;
    constexpr uint32_t B_BYTES = KCH * NPAD * 16;
    constexpr int S = kConvStages;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // TMA destinations on a 1024-byte boundary (the allocation has 1 KB of slack)
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    unsigned char* bsm = smem + S * BOX_ALLOC;
    __shared__ __align__(8) uint64_t bar_full[S], bar_empty[S], bar_accf[2], bar_acce[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int s_fail;
    __shared__ float s_bias[NPAD];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles_w = (a.W + kConvTile - 1) / kConvTile;
    const long long ntiles = (long long)a.N * a.H * tiles_w;
    const int nmine = blockIdx.x < ntiles ? (int)((ntiles - 1 - blockIdx.x) / gridDim.x) + 1 : 0;

    // zero rows, weights (B operand image), barriers, accumulator columns
    for (int s = 0; s < S; s++)
        for (int i = tid; i < kZeroBytes / 16; i += kConvWsThreads)
            reinterpret_cast<uint4*>(smem + s * BOX_ALLOC + BOX_BYTES)[i] = make_uint4(0, 0, 0, 0);
    for (int i = tid; i < (int)(B_BYTES / 16); i += kConvWsThreads) reinterpret_cast<uint4*>(bsm)[i] = a.wpack[i];
    if (tid < NPAD) s_bias[tid] = (a.bias && tid < a.cout) ? a.bias[tid] : 0.f;
    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&bar_full[s], 1);
            mbar_init(&bar_empty[s], 1);
        }
        for (int k = 0; k < 2; k++) {
            mbar_init(&bar_accf[k], 1);
            mbar_init(&bar_acce[k], kConvThreads / 32);
        }
        fence_mbar_init();
        s_fail = 0;
    }
    if (warp == 0) tmem_alloc(&tmem_slot, 64);
    fence_proxy_async();   // generic-proxy writes (zero rows, weights) before tensor-core reads
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    TileWalk walk(blockIdx.x, gridDim.x, tiles_w, a.H);   // the next box, or the epilogue's next tile

    if (warp == kConvEpilogues * kConvThreads / 32 + 1) {
        // ---- loads ----
        const bool leader = elect_one();
        int s = 0, phase = 1, i = 0;   // stage, parity of its previous use
        bool ok = true;
        for (; i < nmine; i++) {
            if (i >= S) ok = __all_sync(0xffffffffu, mbar_wait(&bar_empty[s], (uint32_t)phase));
            if (!ok) break;
            if (leader) {
                mbar_arrive_expect_tx(&bar_full[s], BOX_BYTES);
                tma_load_5d(smem + s * BOX_ALLOC, &tm_in, 0, walk.tw * (kConvTile / PIX) - 1, walk.h - 1, 0, walk.n,
                            &bar_full[s]);
            }
            walk.next();
            if (++s == S) {
                s = 0;
                phase ^= 1;
            }
        }
        if (!ok) {
            s_fail = 1;
            // the copies in flight, before the shared memory is released
            for (int k = max(0, i - S); k < i; k++) mbar_wait(&bar_full[k % S], (uint32_t)((k / S) & 1));
        }
    } else if (warp == kConvEpilogues * kConvThreads / 32) {
        // ---- MMAs ----
        const bool leader = elect_one();
        constexpr uint32_t idesc = umma_idesc(NPAD, false, false), hi = desc_hi(128);
        const uint32_t a0 = desc_lo(smem_u32(smem) + A0, 0), b0 = desc_lo(smem_u32(bsm), NPAD * 16);
        int s = 0, phase = 0, j = 0;
        bool ok = true;
        for (; j < nmine; j++) {
            const int acc = j & 1;
            ok = mbar_wait(&bar_full[s], (uint32_t)phase);
            if (j >= 2) ok = mbar_wait(&bar_acce[acc], (uint32_t)(((j >> 1) - 1) & 1)) && ok;
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            if (leader) {
                const uint32_t alo = a0 + (uint32_t)s * (BOX_ALLOC >> 4);
#pragma unroll
                for (int k = 0; k < KSTEPS; k++) {
                    uint32_t aoff, lbo;
                    if (CH == 4) {
                        const int tap = k >> 1, c0 = (k & 1) * 2;
                        aoff = tap_off(tap, CH, BOXW) + (uint32_t)(c0 * 3 * BOXW * 16);
                        lbo = 3 * BOXW * 16;
                    } else {
                        // tap 9 is the zero rows after the box (from the
                        // operands' shifted start: the same offset minus A0)
                        aoff = tap_off(2 * k, CH, BOXW) - (2 * k >= 9 ? A0 : 0);
                        lbo = tap_off(2 * k + 1, CH, BOXW) - (2 * k + 1 >= 9 ? A0 : 0) - aoff;
                    }
                    umma_bf16(tmem + (uint32_t)(acc * 32), alo + desc_lo(aoff, lbo), hi, b0 + (uint32_t)(2 * k * NPAD),
                              hi, idesc, k > 0 ? 1u : 0u);
                }
                umma_commit(&bar_empty[s]);
                umma_commit(&bar_accf[acc]);
            }
            __syncwarp();
            if (++s == S) {
                s = 0;
                phase ^= 1;
            }
        }
        if (!ok) {
            s_fail = 1;
            // before the shared memory and the accumulator columns are
            // released: the last MMA group (its barrier completes after every
            // earlier group)
            if (j > 0) mbar_wait(&bar_empty[(j - 1) % S], (uint32_t)(((j - 1) / S) & 1));
        }
    } else {
        // ---- epilogue: thread t of the warpgroup owns output pixel w0 + t ----
        const int acc = warp >> 2;   // tiles acc, acc + 2, ..
        if (acc) walk.next();
        for (int j = acc; j < nmine; j += kConvEpilogues) {
            const int n = walk.n, h = walk.h, w = walk.tw * kConvTile + (tid & (kConvThreads - 1));
            walk.next();
            walk.next();
            // the aux input is on its way while the MMAs are
            uint4 act[NPAD / 8];
            float res = 0.f;
            if (w < a.W && a.mode == 2) {
                const long long plane = (long long)a.H * a.W, o = (long long)h * a.W + w;
#pragma unroll
                for (int c = 0; c < NPAD / 8; c++)
                    if (c < a.cout / 8)
                        act[c] = reinterpret_cast<const uint4*>(a.aux)[((long long)n * (a.cout / 8) + c) * plane + o];
            }
            if (w < a.W && a.mode == 1)
                res = reinterpret_cast<const float*>(a.aux)[((long long)n * a.H + h) * a.W + w];
            // (agreed on by the warp: the TMEM load below takes all of it)
            if (!__all_sync(0xffffffffu, mbar_wait(&bar_accf[acc], (uint32_t)((j >> 1) & 1)))) {
                s_fail = 1;
                break;
            }
            tc_fence_after();
            float v[32];
            tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(acc * 32), v);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_acce[acc]);
            if (w < a.W) {
                const long long pix = ((long long)n * a.H + h) * a.W + w;   // pixel index within one channel plane
                const long long plane = (long long)a.H * a.W;
                if (a.mode == 0 || a.mode == 2) {
                    uint4* o = reinterpret_cast<uint4*>(a.out);
                    const int cho = a.cout / 8;
#pragma unroll
                    for (int c = 0; c < NPAD / 8; c++) {
                        if (c >= cho) break;
                        float q[8];
#pragma unroll
                        for (int i = 0; i < 8; i++) q[i] = v[c * 8 + i];
                        const long long idx = ((long long)n * cho + c) * plane + (long long)h * a.W + w;
                        if (a.mode == 0) {
#pragma unroll
                            for (int i = 0; i < 8; i++) q[i] = fmaxf(q[i] + s_bias[c * 8 + i], 0.f);
                        } else {
                            float m[8];
                            unpack_bf16x8(act[c], m);
#pragma unroll
                            for (int i = 0; i < 8; i++) q[i] = m[i] > 0.f ? q[i] : 0.f;
                        }
                        o[idx] = pack_bf16x8(q);
                    }
                } else if (a.mode == 1) {
                    reinterpret_cast<float*>(a.out)[pix] = v[0] + s_bias[0] + res;
                } else {
                    float* o = reinterpret_cast<float*>(a.out);
#pragma unroll
                    for (int c = 0; c < NPAD; c++)   // (constant indices keep v in registers)
                        if (c < a.cout) o[((long long)n * a.cout + c) * plane + (long long)h * a.W + w] = v[c] + s_bias[c];
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && s_fail) atomicExch(a.err, RN_ERR_TIMEOUT);
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, 64);
}

// Shared memory of the weight gradient: per stage the X box as [3 rows][CH
// chunks][box pixels][16 B], a group of ones, then the dY box, padded so that
// the 16 groups of the A operand stay inside the allocation.
template <int CH, int CHO, int PIX>
struct WgradLayout {
    static constexpr uint32_t GROUP = (kConvTile + 2 * PIX) * 16;
    static constexpr uint32_t XBOX = 3 * CH * GROUP;
    static constexpr uint32_t DY = (XBOX + GROUP + 127) & ~127u;
    static constexpr uint32_t DYBOX = CHO * kConvTile * 16;
    static constexpr uint32_t STAGE = (DY + DYBOX + 1023) & ~1023u;
    // the last stage's operands: 16 groups of X from a start up to PIX + 1
    // pixels in, and two dY groups where one is real
    static constexpr uint32_t TAIL = 16 * GROUP + 1024;
    static constexpr uint32_t BYTES = (kWgStages - 1) * STAGE + (STAGE > TAIL ? STAGE : TAIL) + 2048;
};

// ---- weight gradient -------------------------------------------------------------
// D_dx[(dy, ci)][co] = sum_p X[p + (dy, dx)][ci] dY[p][co] for the three dx, both
// operands MN-major (8 pixels x 8 channels per 128-byte core matrix).  The X box
// of a tile lies in shared memory as [row][chunk][pixel][8 channels], so the
// (row, chunk) groups of 8 channels follow one another at one stride and the M
// = 128 rows of the A operand are the 3 dy x CH chunks of 8 channels; the group
// after them is a block of ones, whose rows give the bias gradient sum_p
// dY[p][co].  (The groups after that read whatever follows in shared memory,
// which only feeds accumulator rows that are never read.)  dx moves the operand
// by one pixel.  So a tile takes 3 x 8 MMAs with N = 16 or 32; with the output
// channels as rows (32 of 128 real) and one tap per MMA it took 80.  The issue of
// a tile is one warp's serial stream and bounds the kernel: a 32-channel layer of 8
// images of 512 x 512 took 0.29 ms with 80 MMAs, 0.13 with 24 issued by the lane
// that also loads, and takes 0.076 ms with the loads in their own warp.
// Each CTA writes its partial [32][ncols] to `partial`; conv_wgrad_reduce sums
// them.
struct WgradArgs {
    float* partial;       // [gridDim.x][32][ncols]
    int N, H, W;
    int ncols;
    int* err;
};

// Warp 1 keeps kWgStages tiles' loads (a dY box and an X box each) in flight;
// warp 0 issues the MMAs, and each tile's group commits to its stage's "empty"
// barrier, which the load kWgStages tiles later waits for.
// Boxes take PIX pixels per TMA row as in the forward kernel.
template <int CH, int CHO, int PIX>
__global__ void __launch_bounds__(kConvThreads) conv3x3_wgrad_kernel(const __grid_constant__ CUtensorMap tm_x,
                                                                    const __grid_constant__ CUtensorMap tm_dy,
                                                                    WgradArgs a) {
    using L = WgradLayout<CH, CHO, PIX>;
    constexpr int S = kWgStages;
    constexpr uint32_t A0 = 16 * (PIX - 1);
    constexpr int N = CHO == 4 ? 32 : 16;          // MMA columns per dx
    constexpr int ONES = 3 * CH;                   // first accumulator row / 8 of the bias gradient
    constexpr int BIAS_COL = CH == 4 ? 288 : 80;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    __shared__ __align__(8) uint64_t bar_full[S], bar_empty[S];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int tiles_w = (a.W + kConvTile - 1) / kConvTile;
    const long long ntiles = (long long)a.N * a.H * tiles_w;
    const int nmine = blockIdx.x < ntiles ? (int)((ntiles - 1 - blockIdx.x) / gridDim.x) + 1 : 0;
    // ones after each X box; everything else cleared once (the rows that are
    // never read stay finite)
    for (int i = tid; i < (int)(L::BYTES / 16); i += kConvThreads) {
        const uint32_t o = (uint32_t)i * 16 % L::STAGE;
        const uint32_t v = o >= L::XBOX && o < L::XBOX + L::GROUP ? 0x3F803F80u : 0u;   // bf16 1.0 pairs
        reinterpret_cast<uint4*>(smem)[i] = make_uint4(v, v, v, v);
    }
    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&bar_full[s], 1);
            mbar_init(&bar_empty[s], 1);
        }
        fence_mbar_init();
        s_fail = 0;
    }
    if (warp == 0) tmem_alloc(&tmem_slot, 128);
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    if (warp == 1) {
        // ---- loads ----
        const bool leader = elect_one();
        TileWalk walk(blockIdx.x, gridDim.x, tiles_w, a.H);
        int s = 0, phase = 1, i = 0;   // stage, parity of its previous use
        bool ok = true;
        for (; i < nmine; i++) {
            if (i >= S) ok = __all_sync(0xffffffffu, mbar_wait(&bar_empty[s], (uint32_t)phase));
            if (!ok) break;
            if (leader) {
                unsigned char* st = smem + s * L::STAGE;
                mbar_arrive_expect_tx(&bar_full[s], L::XBOX + L::DYBOX);
                tma_load_5d(st + L::DY, &tm_dy, 0, walk.tw * (kConvTile / PIX), walk.h, 0, walk.n, &bar_full[s]);
                tma_load_5d(st, &tm_x, 0, walk.tw * (kConvTile / PIX) - 1, 0, walk.h - 1, walk.n, &bar_full[s]);
            }
            walk.next();
            if (++s == S) {
                s = 0;
                phase ^= 1;
            }
        }
        if (!ok) {
            s_fail = 1;
            // the copies in flight, before the shared memory is released
            for (int k = max(0, i - S); k < i; k++) mbar_wait(&bar_full[k % S], (uint32_t)((k / S) & 1));
        }
    } else if (warp == 0) {
        // ---- MMAs ----
        const bool leader = elect_one();
        constexpr uint32_t idesc = umma_idesc(N, true, true);
        constexpr uint32_t ahi = desc_hi(L::GROUP), bhi = desc_hi(kConvTile * 16);
        const uint32_t a0 = desc_lo(smem_u32(smem) + A0, 128), b0 = desc_lo(smem_u32(smem) + L::DY, 128);
        int s = 0, phase = 0, j = 0;
        bool ok = true;
        for (; j < nmine; j++) {
            ok = __all_sync(0xffffffffu, mbar_wait(&bar_full[s], (uint32_t)phase));
            if (!ok) break;
            tc_fence_after();
            if (leader) {
                const uint32_t alo = a0 + (uint32_t)s * (L::STAGE >> 4), blo = b0 + (uint32_t)s * (L::STAGE >> 4);
#pragma unroll
                for (int k0 = 0; k0 < kConvTile; k0 += 16)
#pragma unroll
                    for (int dx = 0; dx < 3; dx++)
                        umma_bf16(tmem + (uint32_t)(dx * N), alo + (uint32_t)(k0 + dx), ahi, blo + (uint32_t)k0, bhi,
                                  idesc, k0 > 0 || j > 0 ? 1u : 0u);
                umma_commit(&bar_empty[s]);
            }
            __syncwarp();
            if (++s == S) {
                s = 0;
                phase ^= 1;
            }
        }
        if (!ok) s_fail = 1;
        // the last group completes after every earlier one; where a wait gave
        // up, before the shared memory and the accumulator columns are released
        if (j > 0 && !mbar_wait(&bar_empty[(j - 1) % S], (uint32_t)(((j - 1) / S) & 1))) s_fail = 1;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (!s_fail) {
        // thread = accumulator row (dy, chunk, ci) or a bias row; columns dx N + co
        float* dst = a.partial + (long long)blockIdx.x * 32 * a.ncols;
        const bool any = nmine > 0;
        const int g = tid >> 3, ci = tid & 7;
#pragma unroll
        for (int dx = 0; dx < 3; dx++) {
            float v[32];
            tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(dx * N), v);
            if (g < ONES) {
                const int tap = (g / CH) * 3 + dx;
                const int col = CH == 4 ? tap * 32 + (g % CH) * 8 + ci : (tap / 2) * 16 + (tap % 2) * 8 + ci;
#pragma unroll
                for (int co = 0; co < 32; co++)
                    dst[(long long)co * a.ncols + col] = any && co < 8 * CHO ? v[co] : 0.f;
            } else if (g == ONES && dx == 0) {
#pragma unroll
                for (int co = 0; co < 32; co++) {
                    const float t = any && co < 8 * CHO ? v[co] : 0.f;
                    dst[(long long)co * a.ncols + BIAS_COL + ci] = t;
                    dst[(long long)co * a.ncols + BIAS_COL + 8 + ci] = t;
                }
            } else if (CH == 1 && g == ONES + 1 && dx == 0) {
                // the tenth tap of the 8-channel layout
#pragma unroll
                for (int co = 0; co < 32; co++) dst[(long long)co * a.ncols + 72 + ci] = 0.f;
            }
        }
    }
    if (s_fail && tid == 0) atomicExch(a.err, RN_ERR_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 128);
}

// out[i] = the partials' sum in FP64, in a fixed order: 8 threads take every
// eighth partial, then their sums in turn.  Block (32, 8).
__global__ void __launch_bounds__(256) conv_wgrad_reduce(float* __restrict__ out, const float* __restrict__ partial,
                                                         int nparts, int n) {
    __shared__ double sums[8][32];
    const int i = blockIdx.x * 32 + threadIdx.x;
    double s = 0;
    if (i < n)
        for (int p = threadIdx.y; p < nparts; p += 8) s += partial[(long long)p * n + i];
    sums[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0 && i < n) {
        s = 0;
        for (int k = 0; k < 8; k++) s += sums[k][threadIdx.x];
        out[i] = (float)s;
    }
}

// FP32 image [N][H][W] -> bf16 blocked with 8 channels (channel 0 = image).
__global__ void conv_pack_image(uint4* __restrict__ out, const float* __restrict__ img, const float* __restrict__ sub,
                                float scale, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    q[0] = (img[i] - (sub ? sub[i] : 0.f)) * scale;
    out[i] = pack_bf16x8(q);
}

// ---- host side -----------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// Tensor map over a blocked activation [N][ch][H][W][8] bf16 with the pixels
// taken in groups of `pix` (W a multiple of pix): a box of (8 pix, box_w /
// pix, box_h, ch, 1), each of its rows 16 pix bytes; with `rows_outside` (8 pix,
// box_w / pix, ch, box_h, 1).
static int make_act_map(CUtensorMap* m, const void* base, int N, int ch, int H, int W, int box_w, int box_h,
                        int pix = 1, bool rows_outside = false) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return set_error(RN_ERR_CUDA, "conv: cuTensorMapEncodeTiled unavailable");
    if ((reinterpret_cast<uintptr_t>(base) & 15) != 0) return set_error(RN_ERR_ARG, "conv: activations must be 16-byte aligned");
    const int p = pix;
    cuuint64_t dims[5] = {(cuuint64_t)(8 * p), (cuuint64_t)(W / p), (cuuint64_t)H, (cuuint64_t)ch, (cuuint64_t)N};
    cuuint64_t strides[4] = {(cuuint64_t)(16 * p), (cuuint64_t)W * 16, (cuuint64_t)H * W * 16, (cuuint64_t)ch * H * W * 16};
    cuuint32_t box[5] = {(cuuint32_t)(8 * p), (cuuint32_t)(box_w / p), (cuuint32_t)box_h, (cuuint32_t)ch, 1};
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    if (rows_outside) {   // the box's rows outside its chunks
        std::swap(dims[2], dims[3]);
        std::swap(strides[1], strides[2]);
        std::swap(box[2], box[3]);
    }
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(RN_ERR_ARG, "conv: tensor map encoding failed (" + std::to_string((int)r) + ")");
    return RN_OK;
}

static int sm_count() {
    int dev = 0, n = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
}

template <int CH, int NPAD, int PIX>
static int launch_conv(const CUtensorMap& m, const ConvArgs& a, cudaStream_t st) {
    constexpr int KSTEPS = CH == 4 ? 18 : 5;
    constexpr uint32_t BOX_BYTES = CH * 3 * (kConvTile + 2 * PIX) * 16;
    constexpr uint32_t BOX_ALLOC = (BOX_BYTES + kZeroBytes + 1023) & ~1023u;
    const size_t smem = kConvStages * BOX_ALLOC + 2 * KSTEPS * NPAD * 16 + 1024;
    auto kern = conv3x3_kernel<CH, NPAD, PIX>;
    RN_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    RN_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    const long long ntiles = (long long)a.N * a.H * ((a.W + kConvTile - 1) / kConvTile);
    // as many CTAs per SM as shared memory allows (64 of the SM's 512 TMEM
    // columns each), at most four
    int per_sm = 0, dev = 0, smem_sm = 0;
    RN_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kConvWsThreads, smem));
    RN_CUDA_TRY(cudaGetDevice(&dev));
    RN_CUDA_TRY(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    // (the per-CTA reservation and the static barriers: 2 KB)
    per_sm = std::max(1, std::min(std::max(per_sm, smem_sm / (int)(smem + 2048)), 4));
    const int grid = (int)std::min<long long>(ntiles, (long long)per_sm * sm_count());
    kern<<<grid, kConvWsThreads, smem, st>>>(m, a);
    RN_CUDA_TRY(cudaGetLastError());
    return RN_OK;
}

}  // namespace rn

using namespace rn;

extern "C" int rn_conv3x3(void* d_out, const void* d_in, const void* d_wpack, const float* d_bias, const void* d_aux,
                          int N, int H, int W, int cin, int cout, int mode, int* d_err, void* stream) {
    clear_error();
    if (!d_out || !d_in || !d_wpack || !d_err) return set_error(RN_ERR_ARG, "conv: null argument");
    if (N <= 0 || H <= 0 || W <= 0) return set_error(RN_ERR_ARG, "conv: sizes must be positive");
    if (cin != 8 && cin != 32) return set_error(RN_ERR_ARG, "conv: input channels must be 8 or 32");
    if (mode < 0 || mode > 3) return set_error(RN_ERR_ARG, "conv: bad mode");
    if ((mode == 0 || mode == 2) && cout != 32) return set_error(RN_ERR_ARG, "conv: blocked outputs have 32 channels");
    if (mode == 1 && cout != 1) return set_error(RN_ERR_ARG, "conv: the residual output has one channel");
    if (mode == 3 && cout != 1 && cout != 32) return set_error(RN_ERR_ARG, "conv: cout must be 1 or 32");
    if ((mode == 0 || mode == 1) && !d_bias) return set_error(RN_ERR_ARG, "conv: bias required");
    if ((mode == 1 || mode == 2) && !d_aux) return set_error(RN_ERR_ARG, "conv: aux input required");
    CUtensorMap m;
    ConvArgs a{d_out, reinterpret_cast<const uint4*>(d_wpack), d_bias, d_aux, N, H, W, cout, mode, d_err};
    cudaStream_t st = (cudaStream_t)stream;
    auto run = [&](auto pix) {
        constexpr int P = decltype(pix)::value;
        RN_TRY(make_act_map(&m, d_in, N, cin / 8, H, W, kConvTile + 2 * P, 3, P));
        if (cin == 32) return cout == 32 ? launch_conv<4, 32, P>(m, a, st) : launch_conv<4, 16, P>(m, a, st);
        return cout == 32 ? launch_conv<1, 32, P>(m, a, st) : launch_conv<1, 16, P>(m, a, st);
    };
    if (W % 8 == 0) return run(std::integral_constant<int, 8>{});
    if (W % 2 == 0) return run(std::integral_constant<int, 2>{});
    return run(std::integral_constant<int, 1>{});
}

extern "C" int rn_conv3x3_wgrad_cols(int cin) { return cin == 32 ? 288 + 16 : 80 + 16; }

extern "C" int rn_conv3x3_wgrad(float* d_dw, float* d_partial, size_t partial_bytes, const void* d_x, const void* d_dy,
                                int N, int H, int W, int cin, int cout, int* d_err, void* stream) {
    clear_error();
    if (!d_dw || !d_partial || !d_x || !d_dy || !d_err) return set_error(RN_ERR_ARG, "conv wgrad: null argument");
    if (N <= 0 || H <= 0 || W <= 0) return set_error(RN_ERR_ARG, "conv wgrad: sizes must be positive");
    if ((cin != 8 && cin != 32) || (cout != 8 && cout != 32)) return set_error(RN_ERR_ARG, "conv wgrad: channels 8 or 32");
    const int ncols = rn_conv3x3_wgrad_cols(cin);
    const long long ntiles = (long long)N * H * ((W + kConvTile - 1) / kConvTile);
    const int grid = (int)std::min<long long>(ntiles, (long long)sm_count());
    if (partial_bytes < (size_t)grid * 32 * ncols * sizeof(float))
        return set_error(RN_ERR_ARG, "conv wgrad: partial buffer too small (" + std::to_string((size_t)grid * 32 * ncols * 4) +
                                         " bytes needed)");
    WgradArgs a{d_partial, N, H, W, ncols, d_err};
    cudaStream_t st = (cudaStream_t)stream;
    auto run = [&](auto pix) -> int {
        constexpr int P = decltype(pix)::value;
        CUtensorMap mx, mdy;
        RN_TRY(make_act_map(&mx, d_x, N, cin / 8, H, W, kConvTile + 2 * P, 3, P, true));
        RN_TRY(make_act_map(&mdy, d_dy, N, cout / 8, H, W, kConvTile, 1, P));
        auto launch = [&](auto kern, size_t bytes) -> int {
            const size_t smem = bytes + 1024;
            RN_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            kern<<<grid, kConvThreads, smem, st>>>(mx, mdy, a);
            return RN_OK;
        };
        if (cin == 32 && cout == 32) return launch(conv3x3_wgrad_kernel<4, 4, P>, WgradLayout<4, 4, P>::BYTES);
        if (cin == 32 && cout == 8) return launch(conv3x3_wgrad_kernel<4, 1, P>, WgradLayout<4, 1, P>::BYTES);
        if (cin == 8 && cout == 32) return launch(conv3x3_wgrad_kernel<1, 4, P>, WgradLayout<1, 4, P>::BYTES);
        return set_error(RN_ERR_ARG, "conv wgrad: unsupported channel pair");
    };
    if (W % 8 == 0) RN_TRY(run(std::integral_constant<int, 8>{}));
    else if (W % 2 == 0) RN_TRY(run(std::integral_constant<int, 2>{}));
    else RN_TRY(run(std::integral_constant<int, 1>{}));
    RN_CUDA_TRY(cudaGetLastError());
    const int n = 32 * ncols;
    conv_wgrad_reduce<<<(n + 31) / 32, dim3(32, 8), 0, st>>>(d_dw, d_partial, grid, n);
    RN_CUDA_TRY(cudaGetLastError());
    return RN_OK;
}

extern "C" int rn_conv_pack_image(void* d_out, const float* d_img, const float* d_sub, float scale, int N, int H, int W,
                                  void* stream) {
    clear_error();
    if (!d_out || !d_img) return set_error(RN_ERR_ARG, "conv pack: null argument");
    const long long n = (long long)N * H * W;
    if (n <= 0) return set_error(RN_ERR_ARG, "conv pack: sizes must be positive");
    conv_pack_image<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(reinterpret_cast<uint4*>(d_out), d_img,
                                                                                    d_sub, scale, n);
    RN_CUDA_TRY(cudaGetLastError());
    return RN_OK;
}
