// Kernels of the learned preconditioner's convolutional network (a U-Net
// over [gradient, illumination, Vp, Vs] images), sm_100a:
//
//  * k_conv_kmajor  3x3 convolution (stride 1, zero padding 1) as an
//    implicit GEMM on the tcgen05 tensor cores: M = 128 pixels of one CTA,
//    N = output channels, K = 9 taps x input channels.  Operand tiles are
//    4-D / 3-D TMA boxes of the NHWC activation (shifted by the tap; the
//    zero fill of out-of-range boxes is the padding) and of the weights,
//    in the swizzled K-major layout; a 4-stage mbarrier pipeline feeds one
//    MMA-issuing thread; FP32 accumulators live in tensor memory; the
//    epilogue adds the bias and applies ReLU, or (input gradient) masks by a
//    ReLU output, and stores BF16 NHWC with any channel stride / offset.
//    The same kernel computes the input gradient with the tap-flipped,
//    transposed weights.
//  * k_conv_rows    the same convolution down strips of rows, with the weights
//    resident and each input row used for three output rows; the same bits.
//  * k_conv_wgrad   weight gradient dW[tap][co][ci] = sum_p dz[p][co] x[p+tap][ci]
//    as a GEMM with M = (tap, output channel) pairs, N = input channels,
//    K = pixels, both operands MN-major (channels contiguous in NHWC), split
//    over pixel ranges with FP32 atomic accumulation.
//  * plain kernels for input packing, 2x2 average pooling, nearest 2x
//    upsampling into concatenation buffers, their gradients, the 1x1 output
//    head with its masked mean-square loss, bias gradients, weight packing
//    and the Adam update.
//
// Every mbarrier wait is bounded; a wait that gives up raises an error flag
// that the host reads.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdio>
#include <mutex>
#include <cstring>
#include <string>

#include "../../include/stfwi.h"
#include "../../include/stfwi_nn.h"
#include "tma.cuh"
#include "umma.cuh"

namespace stfwi {
namespace nn {

constexpr int SMS = 148;                 // SMs of a B200, which the grids are cut for
constexpr int CONV_THREADS = 128;
constexpr int STAGES = 4;
constexpr int PIPE_THREADS = 192;         // four epilogue warps (one per quarter of the TMEM lanes), a loader, an issuer
constexpr uint32_t NN_WAIT = 1u << 22;   // mbarrier polls before a wait gives up
constexpr int WG_PIX = 64;                // pixels per k-block of the weight gradient

struct ConvGeo {
    int n, h, w;          // images and spatial size (input = output size)
    int cin, cout;        // channels of the input tensor (contiguous NHWC) and of the output
    int kc;               // input channels per k-block: 16, 32 or 64 (the swizzle atom is 2*kc bytes)
    int bn;               // output channels per CTA (multiple of 16, <= 128)
    int bw, bh;           // pixel box of a CTA, bw * bh = 128
    int y_cstride, y_coff;
    int act;              // 0 none, 1 ReLU
    int m_cstride, m_coff;  // mask (input gradient): multiply by [mask > 0]
    int rows, strips, stages;  // row kernel: output rows of a CTA, strips of them, pipeline stages
};

struct WgradGeo {
    int n, h, w;
    int cout, cin;        // channels of dz (M side) and of x (N side)
    int ae_a, ae_b;       // swizzle atom width in elements along M and along N
    int ca;               // atom columns of dz: cout / ae_a
    int bn;               // input channels per CTA (multiple of ae_b, <= 128)
    int ci_tiles;
    int chunks, chunks_per_split;  // 64-pixel row chunks in total and per CTA
};

__host__ __device__ inline uint32_t tmem_cols_for(int n)
{
    uint32_t c = 32;
    while (c < (uint32_t)n) c <<= 1;
    return c;
}

__device__ __forceinline__ uint8_t *align1024(uint8_t *p)
{
    const uint32_t a = smem_u32(p);
    return p + (((a + 1023u) & ~1023u) - a);
}

__device__ __forceinline__ void store_bf16x16(__nv_bfloat16 *dst, const float (&v)[16])
{
    uint4 q[2];
    __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(q);
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    reinterpret_cast<uint4 *>(dst)[0] = q[0];
    reinterpret_cast<uint4 *>(dst)[1] = q[1];
}

__device__ __forceinline__ void load_bf16x16(const __nv_bfloat16 *src, float (&v)[16])
{
    uint4 q[2];
    q[0] = reinterpret_cast<const uint4 *>(src)[0];
    q[1] = reinterpret_cast<const uint4 *>(src)[1];
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(q);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float2 f = __bfloat1622float2(h[i]);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}

extern __shared__ uint8_t nn_smem[];

// ------------------------------------------------------------------ conv (K-major)

// accumulator row of one pixel -> bias, ReLU or mask, BF16
__device__ __forceinline__ void conv_store(const ConvGeo &g, uint32_t taddr, size_t pix, int n0, bool ok,
                                           const float *__restrict__ bias, const __nv_bfloat16 *__restrict__ mask,
                                           __nv_bfloat16 *__restrict__ y)
{
    for (int c = 0; c < g.bn; c += 16) {
        float v[16];
        tmem_ld16(taddr + (uint32_t)c, v);
        const int ch = n0 + c;
        if (bias) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += __ldg(bias + ch + i);
        }
        if (g.act == 1) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = fmaxf(v[i], 0.f);
        }
        if (mask) {
            float mk[16];
            load_bf16x16(mask + pix * g.m_cstride + g.m_coff + ch, mk);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = mk[i] > 0.f ? v[i] : 0.f;
        }
        if (ok) store_bf16x16(y + pix * g.y_cstride + g.y_coff + ch, v);
    }
}

__global__ void __launch_bounds__(CONV_THREADS, 1)
    k_conv_kmajor(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, ConvGeo g,
                  const float *__restrict__ bias, const __nv_bfloat16 *__restrict__ mask,
                  __nv_bfloat16 *__restrict__ y, int *err)
{
    const uint32_t aw = 2u * g.kc;
    const uint32_t a_bytes = 128u * aw;                      // multiple of 1024
    const uint32_t b_bytes = (uint32_t)g.bn * aw;
    const uint32_t st_bytes = a_bytes + ((b_bytes + 1023u) & ~1023u);
    uint8_t *base = align1024(nn_smem);
    uint64_t *full = reinterpret_cast<uint64_t *>(base + STAGES * st_bytes);
    uint64_t *empty = full + STAGES;
    uint64_t *done = empty + STAGES;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);

    const int warp = threadIdx.x >> 5;
    const int tiles_w = g.w / g.bw, tiles_h = g.h / g.bh;
    int t = blockIdx.x;
    const int w0 = (t % tiles_w) * g.bw;
    t /= tiles_w;
    const int h0 = (t % tiles_h) * g.bh;
    const int img = t / tiles_h;
    const int n0 = blockIdx.y * g.bn;
    const uint32_t ncols = tmem_cols_for(g.bn);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        fence_async_shared();
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(tslot, ncols);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = *tslot;

    const int nkc = g.cin / g.kc;
    const int nk = 9 * nkc;
    const uint32_t layout = umma_layout_for((int)aw);
    const uint32_t sbase = smem_u32(base);

    // warp 0 streams the operand boxes and warp 1 issues the MMAs; a whole warp runs
    // each loop (lane 0 waits and issues, the other lanes wait at the shuffle), so
    // no lane of a working warp spins on the accumulator barrier meanwhile
    const int lane = threadIdx.x & 31;
    if (warp == 0) {
        // producer: one A box (128 shifted pixels x kc channels) and one B box (bn x kc weights) per k-block
        for (int kb = 0; kb < nk; ++kb) {
            int fail = 0;
            if (lane == 0) {
                const int s = kb % STAGES;
                if (kb >= STAGES && !mbar_wait_bounded(&empty[s], ((kb / STAGES) - 1) & 1, NN_WAIT)) {
                    atomicExch(err, 1);
                    fail = 1;
                } else {
                    const int tap = kb / nkc, c0 = (kb % nkc) * g.kc;
                    mbar_arrive_expect_tx(&full[s], a_bytes + b_bytes);
                    tma_load_4d(base + s * st_bytes, &tmX, &full[s], c0, w0 + tap % 3 - 1, h0 + tap / 3 - 1, img);
                    tma_load_3d(base + s * st_bytes + a_bytes, &tmW, &full[s], c0, n0, tap);
                }
            }
            if (__shfl_sync(0xffffffffu, fail, 0)) break;
        }
    } else if (warp == 1) {
        // MMA issuer: kc/16 MMAs (K = 16) per k-block, the K step is +32 bytes inside the swizzle atom
        const uint32_t idesc = umma_idesc_bf16(128, g.bn, 0, 0);
        for (int kb = 0; kb < nk; ++kb) {
            int fail = 0;
            if (lane == 0) {
                const int s = kb % STAGES;
                if (!mbar_wait_bounded(&full[s], (kb / STAGES) & 1, NN_WAIT)) {
                    atomicExch(err, 2);
                    fail = 1;
                } else {
                    tmem_fence_after();
                    const uint32_t sa = sbase + s * st_bytes, sb = sa + a_bytes;
                    for (int k = 0; k < g.kc / 16; ++k) {
                        const uint64_t ad = umma_smem_desc(sa + 32u * k, 16u, 8u * aw, layout);
                        const uint64_t bd = umma_smem_desc(sb + 32u * k, 16u, 8u * aw, layout);
                        umma_bf16(tmem, ad, bd, idesc, (kb | k) != 0);
                    }
                    umma_commit(&empty[s]);
                }
            }
            if (__shfl_sync(0xffffffffu, fail, 0)) break;
        }
        if (lane == 0) umma_commit(done);
        __syncwarp();
    }

    // epilogue: thread m owns accumulator row m (TMEM lane m) = pixel m of the box
    const bool ok = mbar_wait_bounded(done, 0, NN_WAIT);
    if (!ok && (threadIdx.x & 31) == 0) atomicExch(err, 3);
    __syncwarp();
    tmem_fence_after();
    const int m = threadIdx.x;
    const size_t pix = ((size_t)img * g.h + h0 + m / g.bw) * g.w + w0 + m % g.bw;
    conv_store(g, tmem + ((uint32_t)(warp * 32) << 16), pix, n0, ok, bias, mask, y);
    tmem_fence_before();
    __syncthreads();
    if (warp == 0) {
        tmem_fence_after();
        tmem_dealloc(tmem, ncols);
    }
}

// The same convolution down a strip of image rows, 128 pixels wide.  The kernel
// above is bound by its operands' way from L2 into shared memory: nine boxes of
// the input and nine of the weights for each 128 pixels.  Here all weights of the
// CTA's output channels stay in shared memory, and an input row is loaded once for
// each horizontal tap and used for the three output rows that it reaches, whose
// accumulators are in tensor memory (a fourth is being stored meanwhile).  Each
// output row still adds its taps and channels in the order of the kernel above,
// so the results are the same bits.  us at 8 x 160 x 512 (before -> now): 32 ->
// 32 channels 60 -> 33, 96 -> 32 116 -> 88, 32 -> 96 161 -> 74; 64 -> 64
// at 8 x 80 x 256 45 -> 29; 128 -> 384 at 8 x 40 x 128 85 -> 60.
constexpr int ROW_ACC = 4, ROW_STAGES = 8;
template <int KC>
__global__ void __launch_bounds__(PIPE_THREADS, 1)
    k_conv_rows(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, ConvGeo g,
                const float *__restrict__ bias, const __nv_bfloat16 *__restrict__ mask,
                __nv_bfloat16 *__restrict__ y, int *err)
{
    constexpr uint32_t aw = 2u * KC, a_bytes = 128u * aw;
    const uint32_t b_bytes = (uint32_t)g.bn * aw;            // whole swizzle atoms
    const int nkc = g.cin / KC;
    uint8_t *wbase = align1024(nn_smem);
    uint8_t *base = wbase + ((9 * nkc * b_bytes + 1023u) & ~1023u);
    uint64_t *full = reinterpret_cast<uint64_t *>(base + g.stages * a_bytes);
    uint64_t *empty = full + ROW_STAGES;
    uint64_t *wfull = empty + ROW_STAGES;
    uint64_t *done = wfull + 1, *drained = done + ROW_ACC;   // per accumulator: complete; read by the epilogue
    uint64_t *idle = drained + ROW_ACC;                      // every MMA issued is complete
    uint32_t *tslot = reinterpret_cast<uint32_t *>(idle + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_w = g.w / 128;
    int t = blockIdx.x;
    const int w0 = (t % tiles_w) * 128;
    t /= tiles_w;
    const int h0 = (t % g.strips) * g.rows, h1 = min(g.h, h0 + g.rows);
    const int img = t / g.strips;
    const int n0 = blockIdx.y * g.bn;
    const uint32_t ncols = tmem_cols_for(ROW_ACC * g.bn);

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(wfull, 1);
        mbar_init(idle, 1);
        for (int s = 0; s < ROW_ACC; ++s) {
            mbar_init(&done[s], 1);
            mbar_init(&drained[s], 4);
        }
        fence_async_shared();
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(tslot, ncols);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = *tslot;

    // boxes of the strip: input rows h0 - 1 .. h1 (rows outside the image are zeros), for
    // each the three horizontal taps and for each the input-channel blocks
    if (warp == 4) {
        if (lane == 0) {
            mbar_arrive_expect_tx(wfull, 9u * nkc * b_bytes);
            // per (horizontal tap, channel block): vertical taps 2, 1, 0 one below the other
            for (int i = 0; i < 9 * nkc; ++i)
                tma_load_3d(wbase + i * b_bytes, &tmW, wfull, i / 3 % nkc * KC, n0, (2 - i % 3) * 3 + i / 3 / nkc);
            bool ok = true;
            int s = 0, round = 0;
            for (int r = h0 - 1; r <= h1 && ok; ++r)
                for (int dx = 0; dx < 3 && ok; ++dx)
                    for (int c = 0; c < nkc && ok; ++c) {
                        ok = round == 0 || mbar_wait_bounded(&empty[s], (round - 1) & 1, NN_WAIT);
                        if (!ok) break;
                        mbar_arrive_expect_tx(&full[s], a_bytes);
                        tma_load_4d(base + s * a_bytes, &tmX, &full[s], c * KC, w0 + dx - 1, r, img);
                        if (++s == g.stages) {
                            s = 0;
                            ++round;
                        }
                    }
            if (!ok) atomicExch(err, 1);
            // the CTA does not end under a copy in flight, whoever gave up
            mbar_wait_bounded(wfull, 0, NN_WAIT);
            for (int i = 0; i < g.stages; ++i)
                if (i < s || round > 0) mbar_wait_bounded(&full[i], (i < s ? round : round - 1) & 1, NN_WAIT);
        }
        __syncwarp();
    } else if (warp == 5) {
        if (lane == 0) {
            const uint32_t layout = umma_layout_for((int)aw);
            const uint64_t a0 = umma_smem_desc(smem_u32(base), 16u, 8u * aw, layout);
            const uint64_t b0 = umma_smem_desc(smem_u32(wbase), 16u, 8u * aw, layout);
            int s = 0, round = 0;
            bool ok = mbar_wait_bounded(wfull, 0, NN_WAIT);
            for (int r = h0 - 1; r <= h1 && ok; ++r) {
                // output row r + 1 begins here, in the accumulator of row r - 3
                const int first = r + 1 - h0;
                if (r + 1 < h1 && first >= ROW_ACC)
                    ok = mbar_wait_bounded(&drained[first % ROW_ACC], (first / ROW_ACC - 1) & 1, NN_WAIT);
                for (int dx = 0; dx < 3 && ok; ++dx)
                    for (int c = 0; c < nkc && ok; ++c) {
                        ok = mbar_wait_bounded(&full[s], round & 1, NN_WAIT);
                        if (!ok) break;
                        tmem_fence_after();
                        // This row adds to output rows r - 1, r, r + 1 (vertical taps 2, 1, 0), whose
                        // accumulators lie side by side but for the ring's end.  With 64-channel blocks
                        // one MMA serves as many of them as N <= 256 holds, but for row r + 1 where its
                        // accumulator begins (64 -> 64 channels 32 -> 29 us); with smaller blocks the
                        // few K steps of a box do not pay for the longer loop (96 -> 32: 88 -> 97 us).
                        const uint64_t ad = a0 + ((s * a_bytes) >> 4);
                        const uint64_t bd = b0 + (((dx * nkc + c) * 3 * b_bytes) >> 4);
                        const int end = min(h1, r + 2);
                        if constexpr (KC == 64) {
                            for (int o = max(h0, r - 1); o < end;) {
                                const int slot = (o - h0) % ROW_ACC;
                                const bool begins = o == r + 1 && (dx | c) == 0;
                                int m = min(min(end - o, ROW_ACC - slot), 256 / g.bn);
                                if ((dx | c) == 0 && !begins && o + m == r + 2) --m;
                                const uint32_t idesc = umma_idesc_bf16(128, m * g.bn, 0, 0);
                                const uint64_t bo = bd + (((o + 1 - r) * b_bytes) >> 4);
                                // a K step of 16 is +32 bytes inside the swizzle atom (2 in the descriptor)
#pragma unroll
                                for (int k = 0; k < KC / 16; ++k)
                                    umma_bf16(tmem + (uint32_t)(slot * g.bn), ad + 2u * k, bo + 2u * k, idesc,
                                              !begins || k != 0);
                                o += m;
                            }
                        } else {
                            const uint32_t idesc = umma_idesc_bf16(128, g.bn, 0, 0);
#pragma unroll
                            for (int k = 0; k < KC / 16; ++k)
#pragma unroll
                                for (int j = 0; j < 3; ++j) {
                                    const int o = r - 1 + j;
                                    if (o < h0 || o >= end) continue;
                                    umma_bf16(tmem + (uint32_t)(o - h0) % ROW_ACC * g.bn, ad + 2u * k,
                                              bd + ((j * b_bytes) >> 4) + 2u * k, idesc, (dx | c | k) != 0 || j < 2);
                                }
                        }
                        umma_commit(&empty[s]);
                        if (++s == g.stages) {
                            s = 0;
                            ++round;
                        }
                    }
                if (ok && r - 1 >= h0) umma_commit(&done[(r - 1 - h0) % ROW_ACC]);
            }
            if (!ok) atomicExch(err, 2);
            umma_commit(idle);
        }
        __syncwarp();
    } else {
        for (int o = h0; o < h1; ++o) {
            const int k = o - h0, slot = k % ROW_ACC;
            const bool ok = mbar_wait_bounded(&done[slot], (k / ROW_ACC) & 1, NN_WAIT);
            if (!ok && lane == 0) atomicExch(err, 3);
            if (!__all_sync(0xffffffffu, ok)) break;
            tmem_fence_after();
            const size_t pix = ((size_t)img * g.h + o) * g.w + w0 + threadIdx.x;
            conv_store(g, tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(slot * g.bn), pix, n0, true, bias, mask, y);
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&drained[slot]);
        }
    }
    tmem_fence_before();
    __syncthreads();
    if (warp == 0) {
        mbar_wait_bounded(idle, 0, NN_WAIT);   // nor under an MMA
        tmem_fence_after();
        tmem_dealloc(tmem, ncols);
    }
}

// ------------------------------------------------------------------ weight gradient (MN-major)

// Rows of M are (tap, output channel) pairs, an atom column of dz (16, 32 or 64
// channels) each from its own shift of dz: dW[tap] = sum_q dz[q - tap] x[q].  So
// layers of fewer than 128 channels fill their tiles: with one tap a CTA, 32
// channels used a quarter of the rows, and x was read nine times instead of
// three.  What bounds it is the operands' way from L2 into shared memory.  us at
// 8 x 160 x 512 (before -> now): 32 -> 32 channels 209 -> 130, 96 -> 32 660 -> 379; 8 x 40 x
// 128: 128 -> 128 115 -> 52, 384 -> 128 135 -> 103; all 14 layers 2219 -> 1378.
__global__ void __launch_bounds__(PIPE_THREADS, 1)
    k_conv_wgrad(const __grid_constant__ CUtensorMap tmDZ, const __grid_constant__ CUtensorMap tmX, WgradGeo g,
                 float *__restrict__ dw, int *err)
{
    const uint32_t aw_a = 2u * g.ae_a, aw_b = 2u * g.ae_b;
    const int na = 128 / g.ae_a, nb = g.bn / g.ae_b;       // atom columns of a tile along M and along N
    const uint32_t col_a = WG_PIX * aw_a, col_b = WG_PIX * aw_b;  // bytes of one atom column (multiples of 1024)
    const uint32_t a_bytes = na * col_a, b_bytes = nb * col_b;
    const uint32_t st_bytes = a_bytes + b_bytes;
    uint8_t *base = align1024(nn_smem);
    uint64_t *full = reinterpret_cast<uint64_t *>(base + STAGES * st_bytes);
    uint64_t *empty = full + STAGES;
    uint64_t *done = empty + STAGES;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);

    const int warp = threadIdx.x >> 5;
    const int n0 = blockIdx.y * g.bn;
    const int c_begin = blockIdx.x * g.chunks_per_split;
    const int c_end = min(g.chunks, c_begin + g.chunks_per_split);
    const int nk = c_end - c_begin;
    const uint32_t ncols = tmem_cols_for(g.bn);
    // this CTA's atom columns: [a0, a0 + live) of 9 taps x ca.  The tile's columns past the
    // last are not loaded: their accumulator rows hold anything and are not read.
    const int a0 = blockIdx.z * na, live = min(na, 9 * g.ca - a0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
    }
    fence_async_shared();
    __syncwarp();
    if (warp == 0) tmem_alloc(tslot, ncols);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t sbase = smem_u32(base);
    const int wchunks = g.w / WG_PIX;

    const int lane = threadIdx.x & 31;
    if (warp == 4) {
        int s = 0, round = 0;
        for (int kb = 0; kb < nk; ++kb) {
            int fail = 0;
            if (lane == 0) {
                if (round > 0 && !mbar_wait_bounded(&empty[s], (round - 1) & 1, NN_WAIT)) {
                    atomicExch(err, 11);
                    fail = 1;
                } else {
                    int c = c_begin + kb;
                    const int px0 = (c % wchunks) * WG_PIX;
                    c /= wchunks;
                    const int hh = c % g.h, img = c / g.h;
                    mbar_arrive_expect_tx(&full[s], live * col_a + b_bytes);
                    uint8_t *sa = base + s * st_bytes;
                    for (int b = 0; b < nb; ++b)
                        tma_load_4d(sa + a_bytes + b * col_b, &tmX, &full[s], n0 + b * g.ae_b, px0, hh, img);
                    int tap = a0 / g.ca, ch = a0 % g.ca;
                    for (int a = 0; a < live; ++a) {
                        tma_load_4d(sa + a * col_a, &tmDZ, &full[s], ch * g.ae_a, px0 + 1 - tap % 3, hh + 1 - tap / 3,
                                    img);
                        if (++ch == g.ca) {
                            ch = 0;
                            ++tap;
                        }
                    }
                }
            }
            if (__shfl_sync(0xffffffffu, fail, 0)) break;
            if (++s == STAGES) {
                s = 0;
                ++round;
            }
        }
    } else if (warp == 5) {
        // K = 16 pixel rows per MMA: +16 rows of the atom column; LBO = atom column stride, SBO = 8 rows
        const uint32_t idesc = umma_idesc_bf16(128, g.bn, 1, 1);
        const uint32_t la = umma_layout_for((int)aw_a), lb = umma_layout_for((int)aw_b);
        int s = 0, round = 0;
        for (int kb = 0; kb < nk; ++kb) {
            int fail = 0;
            if (lane == 0) {
                if (!mbar_wait_bounded(&full[s], round & 1, NN_WAIT)) {
                    atomicExch(err, 12);
                    fail = 1;
                } else {
                    tmem_fence_after();
                    const uint32_t sa = sbase + s * st_bytes, sb = sa + a_bytes;
#pragma unroll
                    for (int k = 0; k < WG_PIX / 16; ++k) {
                        const uint64_t ad = umma_smem_desc(sa + 16u * aw_a * k, col_a, 8u * aw_a, la);
                        const uint64_t bd = umma_smem_desc(sb + 16u * aw_b * k, col_b, 8u * aw_b, lb);
                        umma_bf16(tmem, ad, bd, idesc, (kb | k) != 0);
                    }
                    umma_commit(&empty[s]);
                }
            }
            if (__shfl_sync(0xffffffffu, fail, 0)) break;
            if (++s == STAGES) {
                s = 0;
                ++round;
            }
        }
        // also where a wait gave up: the accumulators are freed once the MMAs issued are complete
        if (lane == 0) umma_commit(done);
        __syncwarp();
    } else {
        const bool ok = mbar_wait_bounded(done, 0, NN_WAIT);
        if (!ok && lane == 0) atomicExch(err, 13);
        __syncwarp();
        tmem_fence_after();
        const int a = threadIdx.x / g.ae_a, tap = (a0 + a) / g.ca;
        const int co = (a0 + a) % g.ca * g.ae_a + threadIdx.x % g.ae_a;
        float *dst = dw + ((size_t)tap * g.cout + co) * g.cin + n0;
        for (int c = 0; c < g.bn; c += 16) {
            float v[16];
            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
            if (ok && a < live) {
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                    atomicAdd(reinterpret_cast<float4 *>(dst + c + i), make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]));
            }
        }
    }
    tmem_fence_before();
    __syncthreads();
    if (warp == 0) {
        tmem_fence_after();
        tmem_dealloc(tmem, ncols);
    }
}

// ------------------------------------------------------------------ plain kernels

// features [n][4][hd][wd] FP32 (channel scales applied) -> NHWC BF16 [n][h][w][16], zero outside
__global__ void k_pack_input(const float *__restrict__ f, int n, int hd, int wd, int h, int w, float s0, float s1,
                             float s2, float s3, __nv_bfloat16 *__restrict__ x)
{
    const size_t total = (size_t)n * h * w;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < total; p += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)(p % w), i = (int)((p / w) % h), img = (int)(p / ((size_t)w * h));
        float v[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) v[c] = 0.f;
        if (i < hd && j < wd) {
            const size_t plane = (size_t)hd * wd, o = (size_t)img * 4 * plane + (size_t)i * wd + j;
            v[0] = f[o] * s0;
            v[1] = f[o + plane] * s1;
            v[2] = f[o + 2 * plane] * s2;
            v[3] = f[o + 3 * plane] * s3;
        }
        store_bf16x16(x + p * 16, v);
    }
}

// The resampling kernels are memory-bound.  A block takes part of one image
// row (blockIdx.x = image * rows + row, blockIdx.y the part), so the only
// division left is a column's, and a thread moves V channels: 8 (16 bytes)
// where channel counts, strides, offsets and pointers allow it, else one.
// us at batch 8, 160 x 512, one channel a thread before -> 8: upsampling of the
// three levels 382 -> 35, its gradient 123 -> 43, skip gradients 223 -> 56, pooling 69 -> 22.
template <int V> struct Vec {
    float v[V];
    __device__ __forceinline__ void load(const __nv_bfloat16 *p)
    {
        if constexpr (V == 1) {
            v[0] = __bfloat162float(*p);
        } else {
            const uint4 q = *reinterpret_cast<const uint4 *>(p);
            const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&q);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 f = __bfloat1622float2(h[i]);
                v[2 * i] = f.x;
                v[2 * i + 1] = f.y;
            }
        }
    }
    __device__ __forceinline__ void store(__nv_bfloat16 *p) const
    {
        if constexpr (V == 1) {
            *p = __float2bfloat16_rn(v[0]);
        } else {
            uint4 q;
            __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&q);
#pragma unroll
            for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            *reinterpret_cast<uint4 *>(p) = q;
        }
    }
};

// f(row, column, channel) over this block's part of a row of w columns and c channels
template <int V, class F> __device__ __forceinline__ void for_row(int w, int c, F f)
{
    const unsigned cg = c / V, total = (unsigned)w * cg;
    for (unsigned e = blockIdx.y * blockDim.x + threadIdx.x; e < total; e += gridDim.y * blockDim.x) {
        const unsigned j = e / cg;
        f((size_t)blockIdx.x, (int)j, (int)((e - j * cg) * V));
    }
}

// 2x2 average pool of a channel slice: in [n][h][w][in_cstride] at in_coff -> out [n][h/2][w/2][c]
template <int V>
__global__ void k_avgpool2(const __nv_bfloat16 *__restrict__ in, int w, int c, int in_cstride, int in_coff,
                           __nv_bfloat16 *__restrict__ out)
{
    const int wo = w / 2;
    for_row<V>(wo, c, [&](size_t row, int j, int ch) {
        // output rows of all images follow one another, and so do pairs of input rows
        const __nv_bfloat16 *q = in + (2 * row * w + 2 * j) * in_cstride + in_coff + ch;
        Vec<V> a, b, d, e;
        a.load(q);
        b.load(q + in_cstride);
        d.load(q + (size_t)w * in_cstride);
        e.load(q + (size_t)(w + 1) * in_cstride);
#pragma unroll
        for (int k = 0; k < V; ++k) a.v[k] = 0.25f * (a.v[k] + b.v[k] + d.v[k] + e.v[k]);
        a.store(out + (row * wo + j) * c + ch);
    });
}

// gradient of a skip tensor y (a ReLU output stored in a concatenation buffer slice):
// dz = (dcat[slice] + 1/4 dpool[parent]) * [y > 0]  -> contiguous [n][h][w][c]
template <int V>
__global__ void k_skip_grad(const __nv_bfloat16 *__restrict__ dcat, const __nv_bfloat16 *__restrict__ ycat,
                            int cstride, int coff, const __nv_bfloat16 *__restrict__ dpool, int h, int w, int c,
                            __nv_bfloat16 *__restrict__ dz)
{
    for_row<V>(w, c, [&](size_t row, int j, int ch) {
        const size_t p = row * w + j;
        Vec<V> g, y, d;
        const unsigned img = blockIdx.x / (unsigned)h, i = blockIdx.x - img * h;
        g.load(dpool + (((size_t)img * (h / 2) + i / 2) * (w / 2) + j / 2) * c + ch);
        y.load(ycat + p * cstride + coff + ch);
        if (dcat) d.load(dcat + p * cstride + coff + ch);
#pragma unroll
        for (int k = 0; k < V; ++k) {
            float v = 0.25f * g.v[k];
            if (dcat) v += d.v[k];
            g.v[k] = y.v[k] > 0.f ? v : 0.f;
        }
        g.store(dz + p * c + ch);
    });
}

// nearest 2x upsampling of low [n][h][w][c] into channels [0, c) of out [n][2h][2w][out_cstride]; a
// block's row is one of low, whose four copies a thread writes
template <int V>
__global__ void k_upsample2(const __nv_bfloat16 *__restrict__ low, int w, int c, int out_cstride,
                            __nv_bfloat16 *__restrict__ out)
{
    for_row<V>(w, c, [&](size_t row, int j, int ch) {
        Vec<V> v;
        v.load(low + (row * w + j) * c + ch);
        __nv_bfloat16 *q = out + (2 * row * 2 * w + 2 * j) * out_cstride + ch;
        v.store(q);
        v.store(q + out_cstride);
        v.store(q + (size_t)2 * w * out_cstride);
        v.store(q + (size_t)(2 * w + 1) * out_cstride);
    });
}

// gradient through the upsampling into a ReLU output: dz[low] = sum_{2x2} dcat[.., 0:c] * [low > 0]
template <int V>
__global__ void k_upsample2_grad(const __nv_bfloat16 *__restrict__ dcat, int cstride,
                                 const __nv_bfloat16 *__restrict__ low, int w, int c, __nv_bfloat16 *__restrict__ dz)
{
    for_row<V>(w, c, [&](size_t row, int j, int ch) {
        const __nv_bfloat16 *q = dcat + (2 * row * 2 * w + 2 * j) * cstride + ch;
        Vec<V> a, b, d, e, l;
        a.load(q);
        b.load(q + cstride);
        d.load(q + (size_t)2 * w * cstride);
        e.load(q + (size_t)(2 * w + 1) * cstride);
        l.load(low + (row * w + j) * c + ch);
#pragma unroll
        for (int k = 0; k < V; ++k) a.v[k] = l.v[k] > 0.f ? a.v[k] + b.v[k] + d.v[k] + e.v[k] : 0.f;
        a.store(dz + (row * w + j) * c + ch);
    });
}

// 1x1 output head: out[p] = b + sum_c wt[c] y[p][c], y [npix][c] BF16 (c <= 64)
__global__ void k_head_fwd(const __nv_bfloat16 *__restrict__ y, size_t npix, int c, const float *__restrict__ wt,
                           const float *__restrict__ b, float *__restrict__ out)
{
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < npix; p += (size_t)gridDim.x * blockDim.x) {
        float s = b[0];
        for (int k = 0; k < c; k += 16) {
            float v[16];
            load_bf16x16(y + p * c + k, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) s = fmaf(__ldg(wt + k + i), v[i], s);
        }
        out[p] = s;
    }
}

// masked mean-square loss of the head and its gradient:
// L = sum_p wgt[p] (out - target)^2 / norm;  dz[p][c] = dL/dout * wt[c] * [y > 0];
// dwt[c] += sum_p dL/dout y[p][c];  db += sum_p dL/dout;  loss (FP64) += L.
// C channels at compile time: the weight sums stay in registers (with a
// run-time count they lay in local memory: 270 us then, 39 now, at 8 x 160 x 512, 32 channels).
template <int C>   // 0: the loss and db alone
__global__ void k_head_loss_grad(const __nv_bfloat16 *__restrict__ y, size_t npix, const float *__restrict__ wt,
                                 const float *__restrict__ out, const float *__restrict__ target,
                                 const float *__restrict__ wgt, float inv_norm, __nv_bfloat16 *__restrict__ dz,
                                 float *__restrict__ dwt, float *__restrict__ db, double *__restrict__ loss)
{
    __shared__ float s_dw[C ? C : 1];
    __shared__ float s_db;
    __shared__ double s_l;
    for (int i = threadIdx.x; i < C; i += blockDim.x) s_dw[i] = 0.f;
    if (threadIdx.x == 0) {
        s_db = 0.f;
        s_l = 0.0;
    }
    __syncthreads();
    float acc_db = 0.f, acc_dw[C ? C : 1];
    double acc_l = 0.0;
#pragma unroll
    for (int i = 0; i < C; ++i) acc_dw[i] = 0.f;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < npix; p += (size_t)gridDim.x * blockDim.x) {
        const float r = out[p] - target[p];
        const float wp = wgt[p];
        acc_l += (double)wp * r * r * inv_norm;
        const float g = 2.f * wp * r * inv_norm;
        acc_db += g;
#pragma unroll
        for (int k = 0; k < C; k += 16) {
            float v[16], d[16];
            load_bf16x16(y + p * C + k, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                acc_dw[k + i] = fmaf(g, v[i], acc_dw[k + i]);
                d[i] = v[i] > 0.f ? g * __ldg(wt + k + i) : 0.f;
            }
            store_bf16x16(dz + p * C + k, d);
        }
    }
    // over the lanes of a warp, then over the block's warps
#pragma unroll
    for (int i = 0; i < C; ++i) {
        float s = acc_dw[i];
        for (int d = 16; d > 0; d >>= 1) s += __shfl_down_sync(0xffffffffu, s, d);
        if (threadIdx.x % 32 == 0) atomicAdd(&s_dw[i], s);
    }
    for (int d = 16; d > 0; d >>= 1) {
        acc_db += __shfl_down_sync(0xffffffffu, acc_db, d);
        acc_l += __shfl_down_sync(0xffffffffu, acc_l, d);
    }
    if (threadIdx.x % 32 == 0) {
        atomicAdd(&s_db, acc_db);
        atomicAdd(&s_l, acc_l);
    }
    __syncthreads();
    if ((int)threadIdx.x < C) atomicAdd(dwt + threadIdx.x, s_dw[threadIdx.x]);
    if (threadIdx.x == 0) {
        atomicAdd(db, s_db);
        atomicAdd(loss, s_l);
    }
}

// db[c] += sum over pixels of dz[p][c] (NHWC contiguous, c <= 1024): a thread
// keeps to V channels (8, 16 bytes a load, where c and the pointer allow it),
// a block sums its threads' in shared memory.  Four pixels are in flight per
// thread.  us for the 14 layers of a batch of 8: 397 with one 2-byte load in flight a thread, 152 now.
template <int V>
__global__ void k_bias_grad(const __nv_bfloat16 *__restrict__ dz, size_t npix, int c, float *__restrict__ db)
{
    extern __shared__ float s_b[];
    for (int i = threadIdx.x; i < c; i += blockDim.x) s_b[i] = 0.f;
    __syncthreads();
    // threads of the grid in whole pixels: thread t takes channel group t % cg of pixels t / cg, + step, ...
    const unsigned cg = c / V, t = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x / cg;
    const unsigned p0 = t / cg, ch = (t - p0 * cg) * V;
    if (p0 < step) {
        float s[V];
#pragma unroll
        for (int k = 0; k < V; ++k) s[k] = 0.f;
        size_t p = p0;
        for (; p + 3 * (size_t)step < npix; p += 4 * (size_t)step) {
            Vec<V> a[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) a[q].load(dz + (p + q * (size_t)step) * c + ch);
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int k = 0; k < V; ++k) s[k] += a[q].v[k];
        }
        for (; p < npix; p += step) {
            Vec<V> a;
            a.load(dz + p * c + ch);
#pragma unroll
            for (int k = 0; k < V; ++k) s[k] += a.v[k];
        }
#pragma unroll
        for (int k = 0; k < V; ++k) atomicAdd(&s_b[ch + k], s[k]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < c; i += blockDim.x) atomicAdd(db + i, s_b[i]);
}

// FP32 master weights [9][cout][cin] -> BF16 forward layout (same) and input-gradient
// layout wt_t[8 - tap][cin][cout] (taps flipped, channels transposed)
__global__ void k_pack_weights(const float *__restrict__ w32, int cout, int cin, __nv_bfloat16 *__restrict__ wf,
                               __nv_bfloat16 *__restrict__ wt)
{
    const int total = 9 * cout * cin;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const int ci = e % cin, co = (e / cin) % cout, tap = e / (cin * cout);
        const __nv_bfloat16 v = __float2bfloat16_rn(w32[e]);
        wf[e] = v;
        if (wt) wt[((size_t)(8 - tap) * cin + ci) * cout + co] = v;
    }
}

// Adam in the efficient form of Kingma and Ba (bias corrections folded into
// lr_t by the host, eps added to sqrt(v)); gradients cleared afterwards
__global__ void k_adam(float *__restrict__ p, float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       size_t n, float lr_t, float b1, float b2, float eps, float grad_scale)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float gi = g[i] * grad_scale;
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr_t * mi / (sqrtf(vi) + eps);
        g[i] = 0.f;
    }
}

}  // namespace nn
}  // namespace stfwi

// ================================================================== C ABI

using namespace stfwi;
using namespace stfwi::nn;

namespace {

thread_local std::string g_err;

int nn_fail(int code, const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

PFN_cuTensorMapEncodeTiled_v12000 nn_encode_fn()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

CUtensorMapSwizzle swizzle_for(int atom_bytes)
{
    return atom_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                             : atom_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
}

// BF16 tensor of `rank` dims (dims[0] contiguous), box `box`, swizzle matching box[0] * 2 bytes
int encode_bf16(CUtensorMap *m, const void *base, int rank, const cuuint64_t *dims, const cuuint32_t *box)
{
    auto fn = nn_encode_fn();
    if (!fn) return nn_fail(STFWI_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
    cuuint64_t strides[4];
    cuuint64_t s = dims[0] * 2;
    for (int i = 1; i < rank; ++i) {
        strides[i - 1] = s;
        s *= dims[i];
    }
    cuuint32_t es[5] = {1, 1, 1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void *>(base), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for((int)box[0] * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return nn_fail(STFWI_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return STFWI_OK;
}

int check_launch(const char *what)
{
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return nn_fail(STFWI_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    return STFWI_OK;
}

constexpr int NN_MAX_DEVICES = 64;

// one pipeline error flag per device (a kernel writes the flag of its own device)
// the status word of the pipeline waits: a device variable of this module,
// zero when the module loads on a device; its address is looked up once per
// device (under a lock), so no network op allocates or synchronises for it
__device__ int g_nn_err_flag;

int *err_flag()
{
    static std::mutex mu;
    static int *flags[NN_MAX_DEVICES] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NN_MAX_DEVICES) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!flags[dev]) {
        int *f = nullptr;
        if (cudaGetSymbolAddress((void **)&f, g_nn_err_flag) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        flags[dev] = f;
    }
    return flags[dev];
}

// the dynamic shared-memory limit of a kernel is set once per device
template <typename K>
int smem_limit_once(K kern, size_t bytes, bool (&done)[NN_MAX_DEVICES], const char *what)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NN_MAX_DEVICES)
        return nn_fail(STFWI_ERR_CUDA, "%s: no usable current device", what);
    if (!done[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
            return check_launch(what);
        done[dev] = true;
    }
    return STFWI_OK;
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int largest_atom(int c) { return c % 64 == 0 ? 64 : c % 32 == 0 ? 32 : 16; }

// Shared memory per SM is 228 KB (1 KB of it reserved per block); a launch asks for at
// least 228 KB / (512 / tensor-memory columns) so that the CTAs resident on one SM never
// hold more than the SM's 512 tensor-memory columns and tcgen05.alloc never waits.
size_t tmem_floor(int bn)
{
    const size_t per_sm = 233472, ctas = 512 / tmem_cols_for(bn);
    return per_sm / ctas - 1024 + 16;
}

size_t conv_smem(int kc, int bn)
{
    const size_t aw = 2 * kc, a = 128 * aw, b = ((size_t)bn * aw + 1023) & ~(size_t)1023;
    const size_t need = 1024 + STAGES * (a + b) + (2 * STAGES + 1) * 8 + 16;
    return need > tmem_floor(bn) ? need : tmem_floor(bn);
}

size_t wgrad_smem(int bn)
{
    const size_t need = 1024 + STAGES * (size_t)(128 + bn) * WG_PIX * 2 + (2 * STAGES + 1) * 8 + 16;
    return need > tmem_floor(bn) ? need : tmem_floor(bn);
}

// How a convolution is cut into CTAs: strips of rows where the weights of all (or 64 or
// more) output channels fit shared memory and one wave of CTAs has strips of ROWS_MIN
// rows at least, else boxes.  Shorter strips load their two outer rows too often and wait
// for all weights first, narrower pieces read the input again for each: us, boxes against
// strips, 96 -> 32 channels at 1 x 160 x 512 (strips of 3 rows) 21, 23; 192 -> 64 at 8 x 80
// x 256 (32 channels a piece) 87, 117; 128 -> 128 at 8 x 40 x 128 (strips of 5) 41, 29.
constexpr int ROWS_MIN = 4;

struct ConvPlan {
    int bn = 0, rows = 0, strips = 0, stages = 0;   // rows 0: boxes
    size_t smem = 0;
};

ConvPlan conv_plan(int n, int h, int w, int cin, int cout, int kc)
{
    ConvPlan p;
    const size_t sm_smem = 228 * 1024, aw = 2 * kc, a = 128 * aw;
    for (int bn = 128; bn >= 16 && w % 128 == 0; bn -= 16) {
        if (cout % bn || (bn < cout && bn < 64)) continue;
        const size_t fixed = 1024 + ((9 * (cin / kc) * bn * aw + 1023) & ~(size_t)1023) +
                             (2 * ROW_STAGES + 2 + 2 * ROW_ACC) * 8 + 8;
        const size_t cols = tmem_cols_for(ROW_ACC * bn);
        for (int occ = 4; occ >= 1; occ >>= 1) {
            // as many CTAs per SM as tensor memory and shared memory hold
            const size_t cap = occ == 1 ? 227 * 1024 : sm_smem / occ - 1024;
            if (occ * cols > 512 || fixed + 4 * a > cap) continue;
            const double want = (double)occ * SMS / ((double)n * (w / 128) * (cout / bn));
            p.strips = want < 1 ? 1 : want > h ? h : (int)want;
            p.rows = (h + p.strips - 1) / p.strips;
            if (p.rows < ROWS_MIN) break;
            p.strips = (h + p.rows - 1) / p.rows;
            p.bn = bn;
            p.stages = (int)((cap - fixed) / a < (size_t)ROW_STAGES ? (cap - fixed) / a : ROW_STAGES);
            p.smem = fixed + p.stages * a;
            // and no more of them, so that tcgen05.alloc never waits for a CTA of the same kernel
            const size_t least = sm_smem / (512 / cols + 1) - 1024 + 16;
            if (p.smem < least) p.smem = least;
            return p;
        }
    }
    // boxes: all output channels that a tile holds, or fewer while the grid is smaller than the
    // chip (us at batch 1, 128 -> 128 at 40 x 128: 14.8 -> 13.2, 256 -> 256 at 20 x 64: 22 -> 19)
    p = ConvPlan();
    p.bn = cout % 128 == 0 ? 128 : cout % 64 == 0 ? 64 : cout % 32 == 0 ? 32 : 16;
    while (p.bn > 16 && 2.0 * ((double)n * h * w / 128) * (cout / p.bn) <= SMS) p.bn /= 2;
    p.smem = conv_smem(kc, p.bn);
    return p;
}

int conv_common(const void *x, int n, int h, int w, int cin, const void *wt, int cout, const float *bias, int act,
                const void *mask, int m_cstride, int m_coff, void *y, int y_cstride, int y_coff, cudaStream_t st)
{
    if (n <= 0 || h <= 0 || w <= 0) return nn_fail(STFWI_ERR_INVALID, "conv: empty image batch");
    if (cin % 16 || cout % 16 || cin <= 0 || cout <= 0)
        return nn_fail(STFWI_ERR_INVALID, "conv: channel counts must be positive multiples of 16 (%d, %d)", cin, cout);
    const int bw = w >= 128 ? 128 : w;
    if (w % bw || 128 % bw || h % (128 / bw))
        return nn_fail(STFWI_ERR_INVALID, "conv: %dx%d does not tile into 128-pixel boxes", h, w);
    if (y_cstride % 8 || y_coff % 8 || y_coff + cout > y_cstride)
        return nn_fail(STFWI_ERR_INVALID, "conv: output channel stride/offset must be multiples of 8 and hold cout");
    if (mask && (m_cstride % 8 || m_coff % 8 || m_coff + cout > m_cstride))
        return nn_fail(STFWI_ERR_INVALID, "conv: mask channel stride/offset");
    if (!aligned16(x) || !aligned16(wt) || !aligned16(y) || (mask && !aligned16(mask)))
        return nn_fail(STFWI_ERR_INVALID, "conv: tensors must be 16-byte aligned");
    ConvGeo g{};
    g.n = n; g.h = h; g.w = w; g.cin = cin; g.cout = cout;
    g.kc = largest_atom(cin);
    const ConvPlan plan = conv_plan(n, h, w, cin, cout, g.kc);
    g.bn = plan.bn;
    g.rows = plan.rows; g.strips = plan.strips; g.stages = plan.stages;
    g.bw = bw; g.bh = 128 / bw;
    g.y_cstride = y_cstride; g.y_coff = y_coff; g.act = act;
    g.m_cstride = m_cstride; g.m_coff = m_coff;
    CUtensorMap tx, tw;
    const cuuint64_t dx[4] = {(cuuint64_t)cin, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
    const cuuint32_t bx[4] = {(cuuint32_t)g.kc, (cuuint32_t)g.bw, (cuuint32_t)g.bh, 1};
    int rc = encode_bf16(&tx, x, 4, dx, bx);
    if (rc) return rc;
    const cuuint64_t dw[3] = {(cuuint64_t)cin, (cuuint64_t)cout, 9};
    const cuuint32_t bwx[3] = {(cuuint32_t)g.kc, (cuuint32_t)g.bn, 1};
    rc = encode_bf16(&tw, wt, 3, dw, bwx);
    if (rc) return rc;
    int *err = err_flag();
    if (!err) return nn_fail(STFWI_ERR_CUDA, "conv: the error flag of this device could not be looked up");
    static bool attr[4][NN_MAX_DEVICES] = {};
    auto go = [&](auto kern, size_t limit, bool (&done)[NN_MAX_DEVICES], dim3 grid, int threads) {
        const int e = smem_limit_once(kern, limit, done, "conv: shared-memory attribute");
        if (e) return e;
        kern<<<grid, threads, plan.smem, st>>>(tx, tw, g, bias, static_cast<const __nv_bfloat16 *>(mask),
                                               static_cast<__nv_bfloat16 *>(y), err);
        return check_launch("convolution");
    };
    const unsigned groups = (unsigned)(cout / g.bn);
    if (!g.rows)
        return go(k_conv_kmajor, conv_smem(64, 128), attr[0],
                  dim3((unsigned)((size_t)n * (h / g.bh) * (w / g.bw)), groups), CONV_THREADS);
    const dim3 grid((unsigned)((size_t)n * g.strips * (w / 128)), groups);
    return g.kc == 64   ? go(k_conv_rows<64>, 227 * 1024, attr[1], grid, PIPE_THREADS)
           : g.kc == 32 ? go(k_conv_rows<32>, 227 * 1024, attr[2], grid, PIPE_THREADS)
                        : go(k_conv_rows<16>, 227 * 1024, attr[3], grid, PIPE_THREADS);
}

unsigned blocks_for(size_t n, int threads)
{
    size_t b = (n + threads - 1) / threads;
    return (unsigned)(b < 1 ? 1 : b > 4 * SMS * 8 ? 4 * SMS * 8 : b);
}

// grid of a row kernel: rows x parts of a row of `per_row` thread items, about four items a thread
dim3 row_grid(size_t rows, size_t per_row)
{
    const size_t parts = (per_row + 1023) / 1024;
    return dim3((unsigned)rows, (unsigned)(parts < 1 ? 1 : parts > 64 ? 64 : parts));
}

// may a row kernel move 8 channels a thread
bool by8(int c, int cstride, int coff, const void *a, const void *b, const void *d = nullptr, const void *e = nullptr)
{
    return c % 8 == 0 && cstride % 8 == 0 && coff % 8 == 0 && aligned16(a) && aligned16(b) && aligned16(d) && aligned16(e);
}

}  // namespace

extern "C" {

const char *stfwi_nn_last_error(void) { return g_err.c_str(); }

int stfwi_nn_check(void *stream)
{
    int *err = err_flag();
    if (!err) return nn_fail(STFWI_ERR_CUDA, "the error flag of this device could not be looked up");
    int v = 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemcpyAsync(&v, err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return check_launch("stfwi_nn_check");
    if (v) {
        cudaMemsetAsync(err, 0, sizeof(int), st);
        cudaStreamSynchronize(st);
        return nn_fail(STFWI_ERR_CUDA, "a tensor-core pipeline wait gave up (code %d)", v);
    }
    return STFWI_OK;
}

int stfwi_nn_conv3x3(const void *x, int n, int h, int w, int cin, const void *wt, int cout, const float *bias,
                     int relu, void *y, int y_cstride, int y_coff, void *stream)
{
    return conv_common(x, n, h, w, cin, wt, cout, bias, relu ? 1 : 0, nullptr, 0, 0, y, y_cstride, y_coff,
                       static_cast<cudaStream_t>(stream));
}

int stfwi_nn_conv3x3_dgrad(const void *dz, int n, int h, int w, int cout, const void *wt_t, int cin,
                           const void *mask, int m_cstride, int m_coff, void *dx, void *stream)
{
    return conv_common(dz, n, h, w, cout, wt_t, cin, nullptr, 0, mask, m_cstride, m_coff, dx, cin, 0,
                       static_cast<cudaStream_t>(stream));
}

int stfwi_nn_conv3x3_wgrad(const void *x, const void *dz, int n, int h, int w, int cin, int cout, float *dw,
                           void *stream)
{
    if (n <= 0 || h <= 0 || w <= 0) return nn_fail(STFWI_ERR_INVALID, "wgrad: empty image batch");
    if (cin % 16 || cout % 16 || cin <= 0 || cout <= 0)
        return nn_fail(STFWI_ERR_INVALID, "wgrad: channel counts must be positive multiples of 16");
    if (w % WG_PIX) return nn_fail(STFWI_ERR_INVALID, "wgrad: width must be a multiple of %d", WG_PIX);
    if (!aligned16(x) || !aligned16(dz) || !aligned16(dw))
        return nn_fail(STFWI_ERR_INVALID, "wgrad: tensors must be 16-byte aligned");
    WgradGeo g{};
    g.n = n; g.h = h; g.w = w; g.cout = cout; g.cin = cin;
    g.ae_a = largest_atom(cout);
    g.ca = cout / g.ae_a;
    g.bn = cin % 128 == 0 ? 128 : cin % 64 == 0 ? 64 : cin % 32 == 0 ? 32 : 16;
    g.ae_b = g.bn >= 64 ? 64 : g.bn;
    g.ci_tiles = cin / g.bn;
    const int na = 128 / g.ae_a, groups = (9 * g.ca + na - 1) / na;
    g.chunks = n * h * (w / WG_PIX);
    // The tensor cores cut the low bits of a sum off, so the length of the sums decides how
    // far a gradient is from FP64's: they stay as long as with one tap, 128 output channels
    // and bn input channels a CTA and four CTAs per SM, whatever share of the rows is filled.
    // (Three tiles a CTA and one CTA per SM took 833 us in all, but moved gradients of 12
    // images of 320 x 1024 by up to 8e-5 of their norm; this keeps them within 8e-7.)
    const int tiles = 9 * ((cout + 127) / 128) * g.ci_tiles;
    int splits = (4 * SMS + tiles - 1) / tiles;
    if (splits > g.chunks) splits = g.chunks;
    if (splits < 1) splits = 1;
    g.chunks_per_split = (g.chunks + splits - 1) / splits;
    splits = (g.chunks + g.chunks_per_split - 1) / g.chunks_per_split;
    CUtensorMap ta, tb;
    const cuuint64_t da[4] = {(cuuint64_t)cout, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
    const cuuint32_t ba[4] = {(cuuint32_t)g.ae_a, WG_PIX, 1, 1};
    int rc = encode_bf16(&ta, dz, 4, da, ba);
    if (rc) return rc;
    const cuuint64_t db[4] = {(cuuint64_t)cin, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
    const cuuint32_t bb[4] = {(cuuint32_t)g.ae_b, WG_PIX, 1, 1};
    rc = encode_bf16(&tb, x, 4, db, bb);
    if (rc) return rc;
    int *err = err_flag();
    if (!err) return nn_fail(STFWI_ERR_CUDA, "wgrad: the error flag of this device could not be looked up");
    static bool attr[NN_MAX_DEVICES] = {};
    rc = smem_limit_once(k_conv_wgrad, wgrad_smem(128), attr, "wgrad: shared-memory attribute");
    if (rc) return rc;
    const dim3 grid((unsigned)splits, (unsigned)g.ci_tiles, (unsigned)groups);
    k_conv_wgrad<<<grid, PIPE_THREADS, wgrad_smem(g.bn), static_cast<cudaStream_t>(stream)>>>(ta, tb, g, dw, err);
    return check_launch("k_conv_wgrad");
}

int stfwi_nn_pack_input(const float *feat, int n, int hd, int wd, int h, int w, const float *scale4, void *x,
                        void *stream)
{
    if (hd > h || wd > w || n <= 0) return nn_fail(STFWI_ERR_INVALID, "pack_input: sizes");
    const size_t total = (size_t)n * h * w;
    k_pack_input<<<blocks_for(total, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        feat, n, hd, wd, h, w, scale4[0], scale4[1], scale4[2], scale4[3], static_cast<__nv_bfloat16 *>(x));
    return check_launch("k_pack_input");
}

int stfwi_nn_avgpool2(const void *in, int n, int h, int w, int c, int in_cstride, int in_coff, void *out,
                      void *stream)
{
    if (h % 2 || w % 2) return nn_fail(STFWI_ERR_INVALID, "avgpool2: odd size");
    const bool v8 = by8(c, in_cstride, in_coff, in, out);
    const size_t rows = (size_t)n * (h / 2);
    if (n > 0 && h > 0 && w > 0 && c > 0)
        (v8 ? k_avgpool2<8> : k_avgpool2<1>)<<<row_grid(rows, (size_t)(w / 2) * c / (v8 ? 8 : 1)), 256, 0,
                                               static_cast<cudaStream_t>(stream)>>>(
            static_cast<const __nv_bfloat16 *>(in), w, c, in_cstride, in_coff, static_cast<__nv_bfloat16 *>(out));
    return check_launch("k_avgpool2");
}

int stfwi_nn_skip_grad(const void *dcat, const void *ycat, int cstride, int coff, const void *dpool, int n, int h,
                       int w, int c, void *dz, void *stream)
{
    const bool v8 = by8(c, cstride, coff, dcat, ycat, dpool, dz);
    const size_t rows = (size_t)n * h;
    if (n > 0 && h > 0 && w > 0 && c > 0)
        (v8 ? k_skip_grad<8> : k_skip_grad<1>)<<<row_grid(rows, (size_t)w * c / (v8 ? 8 : 1)), 256, 0,
                                                 static_cast<cudaStream_t>(stream)>>>(
            static_cast<const __nv_bfloat16 *>(dcat), static_cast<const __nv_bfloat16 *>(ycat), cstride, coff,
            static_cast<const __nv_bfloat16 *>(dpool), h, w, c, static_cast<__nv_bfloat16 *>(dz));
    return check_launch("k_skip_grad");
}

int stfwi_nn_upsample2(const void *low, int n, int h, int w, int c, int out_cstride, void *out, void *stream)
{
    const bool v8 = by8(c, out_cstride, 0, low, out);
    const size_t rows = (size_t)n * h;
    if (n > 0 && h > 0 && w > 0 && c > 0)
        (v8 ? k_upsample2<8> : k_upsample2<1>)<<<row_grid(rows, (size_t)w * c / (v8 ? 8 : 1)), 256, 0,
                                                 static_cast<cudaStream_t>(stream)>>>(
            static_cast<const __nv_bfloat16 *>(low), w, c, out_cstride, static_cast<__nv_bfloat16 *>(out));
    return check_launch("k_upsample2");
}

int stfwi_nn_upsample2_grad(const void *dcat, int cstride, const void *low, int n, int h, int w, int c, void *dz,
                            void *stream)
{
    const bool v8 = by8(c, cstride, 0, dcat, low, dz);
    const size_t rows = (size_t)n * h;
    if (n > 0 && h > 0 && w > 0 && c > 0)
        (v8 ? k_upsample2_grad<8> : k_upsample2_grad<1>)<<<row_grid(rows, (size_t)w * c / (v8 ? 8 : 1)), 256, 0,
                                                           static_cast<cudaStream_t>(stream)>>>(
            static_cast<const __nv_bfloat16 *>(dcat), cstride, static_cast<const __nv_bfloat16 *>(low), w, c,
            static_cast<__nv_bfloat16 *>(dz));
    return check_launch("k_upsample2_grad");
}

int stfwi_nn_head(const void *y, size_t npix, int c, const float *wt, const float *b, float *out, void *stream)
{
    if (c % 16 || c > 64) return nn_fail(STFWI_ERR_INVALID, "head: channels must be a multiple of 16, <= 64");
    k_head_fwd<<<blocks_for(npix, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16 *>(y), npix, c, wt, b, out);
    return check_launch("k_head_fwd");
}

int stfwi_nn_head_loss_grad(const void *y, size_t npix, int c, const float *wt, const float *out,
                            const float *target, const float *wgt, float inv_norm, void *dz, float *dwt, float *db,
                            double *loss, void *stream)
{
    if (c % 16 || c > 64) return nn_fail(STFWI_ERR_INVALID, "head: channels must be a multiple of 16, <= 64");
    unsigned blocks = blocks_for(npix, 256);
    if (blocks > 8 * SMS) blocks = 8 * SMS;
    auto go = [&](auto kern) {
        kern<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const __nv_bfloat16 *>(y), npix, wt, out, target, wgt, inv_norm, static_cast<__nv_bfloat16 *>(dz),
            dwt, db, loss);
    };
    switch (c) {
    default: go(k_head_loss_grad<0>); break;
    case 16: go(k_head_loss_grad<16>); break;
    case 32: go(k_head_loss_grad<32>); break;
    case 48: go(k_head_loss_grad<48>); break;
    case 64: go(k_head_loss_grad<64>); break;
    }
    return check_launch("k_head_loss_grad");
}

int stfwi_nn_bias_grad(const void *dz, size_t npix, int c, float *db, void *stream)
{
    if (c <= 0 || c > 1024) return nn_fail(STFWI_ERR_INVALID, "bias_grad: channel count %d", c);
    const int threads = 256;
    const bool v8 = c % 8 == 0 && aligned16(dz);
    unsigned blocks = blocks_for(npix * c / (v8 ? 128 : 64), threads);
    if (blocks > 8 * SMS) blocks = 8 * SMS;
    // at least one whole pixel's channels among the threads of the grid
    if (blocks * threads < (unsigned)c) blocks = (c + threads - 1) / threads;
    (v8 ? k_bias_grad<8> : k_bias_grad<1>)<<<blocks, threads, c * sizeof(float), static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16 *>(dz), npix, c, db);
    return check_launch("k_bias_grad");
}

int stfwi_nn_pack_weights(const float *w32, int cout, int cin, void *wf, void *wt, void *stream)
{
    const int total = 9 * cout * cin;
    k_pack_weights<<<blocks_for(total, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        w32, cout, cin, static_cast<__nv_bfloat16 *>(wf), static_cast<__nv_bfloat16 *>(wt));
    return check_launch("k_pack_weights");
}

int stfwi_nn_adam(float *p, float *g, float *m, float *v, size_t n, float lr_t, float b1, float b2, float eps,
                  float grad_scale, void *stream)
{
    k_adam<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(p, g, m, v, n, lr_t, b1, b2, eps,
                                                                            grad_scale);
    return check_launch("k_adam");
}

}  // extern "C"
