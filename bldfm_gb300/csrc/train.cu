// One training step of the surrogate MLP in three launches.
//
//  1. mlp_step_kernel: each CTA takes pairs of 128-sample tiles through the
//     whole network and back.  The activations of a layer never leave shared
//     memory on their way to the next GEMM (they are its A operand, written in
//     place of the previous ones); the accumulators stay in tensor memory.
//     The two tiles are out of step: one's epilogue runs under the other's
//     MMAs.  What the weight gradients need (activations, dZ, inputs) is
//     written once, as the bf16 tiles it is multiplied in.
//  2. mlp_grad_kernel: dW = dZ^T H over a range of samples per CTA.  Both
//     operands are the tiles as written (sample rows, 8-feature core
//     matrices), read as MN-major operands, so nothing is transposed; a CTA
//     holds the whole 256 x 256 sum in its 512 tensor-memory columns.
//  3. mlp_update_kernel: the partial sums in a fixed order (no atomics: a
//     step gives the same bits every time), Adam and the bf16 weight blocks.
//
// Bounds at 65,536 samples: 77 GFLOP of MMA (41 us at the measured BF16 peak);
// 0.67 GB through L2 and HBM (activations, dZ, gelu', each written and read
// once; 100 us at the HBM rate); and in the step kernel the CUDA cores: 16
// packed FP32 operations and four tanh per two activations, 3.4 us for every
// layer of every tile pair (55 us in all).  Measured: step 144 us, gradients
// 53 us, update 16 us; the step kernel's 96 registers a thread (18 warps) spill
// some 40 words.  The layer-by-layer form before it (one launch per
// GEMM, transposed copies of every operand, FP32 activations through HBM,
// shuffled column sums, an atomic per gradient element) took 1,280 us.
#include "devattr.h"
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "mlp_common.cuh"
#include "tc.cuh"
#include "train.h"

namespace {

const int TILE = 128;                      // samples per tile (tensor-memory lanes)
const int TILE_ELEMS = TILE * MLP_H;       // bf16 elements of an activation tile
const uint32_t TILE_BYTES = TILE_ELEMS * 2;
const int XP_COLS = 32;                    // columns of the input pieces: 3 x 8, ones, zeros
const uint32_t CHUNK_BYTES = MLP_H * MLP_KC * 2;
const int NCHUNK = MLP_H / MLP_KC;
const int PB_H = MLP_H * MLP_H + MLP_H;    // one hidden layer's partial: Wt, b
const int PB_0 = MLP_IN * MLP_H + MLP_H;   // the input layer's: W0, b0
const int PB_O = 1032;                     // the output layer's: W4, b4, loss, padding

__device__ __forceinline__ uint4 pack8(const float *v)
{
    return make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                      pack_bf16x2(v[6], v[7]));
}

// h = gelu(z) and g = gelu'(z) for two values.  h rounds as gelu_f does; g takes
// its tanh's argument as c (z + (a z^2) z), rounded after each of these, and h's
// as z (c + (c a) z^2): the bf16 roundings downstream turn one changed last bit
// in 10^4 into a changed activation, which moves a small batch's gradient by 5e-5
__device__ __forceinline__ void gelu_both(float2 z, float2 &h, float2 &g)
{
    auto c2 = [](float v) { return make_float2(v, v); };
    const float2 z2 = __fmul2_rn(z, z), hz = __fmul2_rn(c2(0.5f), z);
    const float2 u = __fmul2_rn(z, __ffma2_rn(c2(GELU_C * GELU_A), z2, c2(GELU_C)));
    h = __ffma2_rn(hz, make_float2(tanh_approx(u.x), tanh_approx(u.y)), hz);
    const float2 v = __fmul2_rn(c2(GELU_C), __ffma2_rn(__fmul2_rn(c2(GELU_A), z2), z, z));
    const float2 t = make_float2(tanh_approx(v.x), tanh_approx(v.y));
    const float2 s = __ffma2_rn(make_float2(-t.x, -t.y), t, c2(1.f));
    const float2 du = __ffma2_rn(c2(3.0f * GELU_A), z2, c2(1.f));
    g = __ffma2_rn(c2(0.5f), __fadd2_rn(t, c2(1.f)), __fmul2_rn(__fmul2_rn(__fmul2_rn(hz, s), c2(GELU_C)), du));
}

// a row of four of the caller's floats, which may sit at any 4-byte address
__device__ __forceinline__ float4 load_row4(const float *__restrict__ p, bool aligned)
{
    if (aligned) return __ldg((const float4 *)p);
    return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}

__device__ __forceinline__ void lds8(float *v, const float *p)
{
    const float4 a = *(const float4 *)p, b = *(const float4 *)(p + 4);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}

struct StepArgs {
    const float *X, *T, *w, *P;
    const uint16_t *Wf[3], *Wb[3];
    MlpTrainBuf b;
    int pairs;     // pairs of tiles
    bool aligned;  // X, T and w start on 16-byte boundaries
    float inv_n;
    int *err;
};

// Warps 8 t .. 8 t + 7 own tile t of the pair (thread = sample row, half the
// columns: tensor-memory lanes allow a warp one quarter of the rows); warp 16
// issues every MMA, warp 17 every weight copy.
const int STEP_WARPS = 18;
const int STEP_THREADS = STEP_WARPS * 32;
const int RING = 3;  // weight chunks in flight
// shared memory: two A tiles, the ring, the dW4 staging (tile, column half:
// 128 rows x 16 columns; before that the outputs y and dY), the biases of all
// layers and W4
const int STG = 16 * TILE * 4;
const int OFF_RING = 2 * (int)(TILE * MLP_H * 2);
const int OFF_STG = OFF_RING + RING * (int)(MLP_H * MLP_KC * 2);
const int OFF_BIAS = OFF_STG + 4 * STG;
const int OFF_W4 = OFF_BIAS + 4 * MLP_H * 4;
const int STEP_SMEM = OFF_W4 + MLP_H * MLP_OUT * 4;
const int NGEMM = 6;  // the hidden layers forward, then back

// One step of a sum shared out over lanes: the lane with bit 4 W set keeps
// entries W .. 2 W - 1 of the pair's sums, the other 0 .. W - 1 (in s[0..W))
template <int W>
__device__ __forceinline__ void share(float2 (&s)[8], int lane, std::integral_constant<int, W>)
{
    const bool up = (lane & (4 * W)) != 0;
#pragma unroll
    for (int k = 0; k < W; ++k) {
        const float2 keep = up ? s[k + W] : s[k], give = up ? s[k] : s[k + W];
        s[k].x = keep.x + __shfl_xor_sync(0xffffffffu, give.x, 4 * W);
        s[k].y = keep.y + __shfl_xor_sync(0xffffffffu, give.y, 4 * W);
    }
}

__global__ void __launch_bounds__(STEP_THREADS, 1) mlp_step_kernel(const StepArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    // ring slots filled / free again; per tile: A written, accumulator complete
    __shared__ uint64_t full[RING], empty[RING], ready[2], done[2], drain;
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float *s_bias = (float *)(smem + OFF_BIAS);
    float4 *s_w4 = (float4 *)(smem + OFF_W4);
    if (warp == 16) tc_tmem_alloc(&tmem_slot, 2 * MLP_H);
    if (tid == 0) {
        for (int i = 0; i < RING; ++i) {
            tc_mbar_init(&full[i], 1);
            tc_mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc_mbar_init(&ready[i], 8);
            tc_mbar_init(&done[i], 1);
        }
        tc_mbar_init(&drain, 1);
        tc_fence_init();
    }
    for (int i = tid; i < 4 * MLP_H; i += STEP_THREADS) {
        const int j = i >> 8, f = i & 255;
        s_bias[i] = a.P[(j == 0 ? MLP_OFF_B0 : MLP_OFF_B(j)) + f];
        ((float *)s_w4)[i] = a.P[MLP_OFF_W4 + i];
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int npairs = (a.pairs - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    bool ok = true;

    if (warp == 17) {
        // ---- weight copies: both tiles' GEMMs in the order warp 16 runs them ----
        uint32_t q = 0;
        for (int p = 0; p < npairs && ok; ++p)
#pragma unroll 1
            for (int g = 0; g < NGEMM && ok; ++g) {
                const uint16_t *w = g < 3 ? a.Wf[g] : a.Wb[5 - g];
#pragma unroll 1
                for (int c2 = 0; c2 < 2 * NCHUNK; ++c2, ++q) {
                    const int c = c2 % NCHUNK, s = (int)(q % RING);
                    if (q >= RING) ok = tc_mbar_wait(&empty[s], (q / RING - 1) & 1);
                    if (!ok) break;
                    tc_load_warp(smem + OFF_RING + s * CHUNK_BYTES, w + (size_t)c * MLP_H * MLP_KC, CHUNK_BYTES,
                                 CHUNK_BYTES, &full[s]);
                }
            }
        // every copy has landed before the block's memory is given back
        for (uint32_t k = q > RING ? q - RING : 0; k < q; ++k) tc_mbar_wait(&full[k % RING], (k / RING) & 1);
    } else if (warp == 16) {
        // ---- MMAs: layer by layer, tile 0 then tile 1 ----
        uint32_t q = 0, nready = 0;
        const uint32_t idesc = tc_idesc_bf16(TILE, MLP_H);
        for (int p = 0; p < npairs && ok; ++p)
#pragma unroll 1
            for (int g = 0; g < NGEMM && ok; ++g, ++nready) {
#pragma unroll 1
                for (int t = 0; t < 2 && ok; ++t) {
                    ok = tc_mbar_wait(&ready[t], nready & 1);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t da = tc_desc(tc_smem(smem + t * TILE_BYTES), 128, (MLP_H / 8) * 128);
                    const uint32_t d = tmem + (uint32_t)(t * MLP_H);
#pragma unroll 1
                    for (int c = 0; c < NCHUNK; ++c, ++q) {
                        const int s = (int)(q % RING);
                        ok = tc_mbar_wait(&full[s], (q / RING) & 1);
                        if (!ok) break;
                        tc_fence_after();
                        const uint64_t db = tc_desc(tc_smem(smem + OFF_RING + s * CHUNK_BYTES), 128, (MLP_KC / 8) * 128);
                        // 16 K columns further: two core matrices, 256 bytes (descriptor units of 16)
#pragma unroll
                        for (int ks = 0; ks < MLP_KC / 16; ++ks)
                            tc_mma_warp(d, da + (uint64_t)((c * (MLP_KC / 16) + ks) * 16), db + (uint64_t)(ks * 16), idesc,
                                        (c > 0 || ks > 0) ? 1u : 0u);
                        tc_commit_warp(&empty[s]);
                    }
                    tc_commit_warp(&done[t]);
                }
            }
    } else {
        // ---- epilogues ----
        const int t = warp >> 3, half = (warp >> 2) & 1, row = (warp & 3) * 32 + lane;
        const int bar_tile = 1 + t, bar_half = 3 + t * 2 + half;
        uint16_t *sA = (uint16_t *)(smem + t * TILE_BYTES);
        unsigned char *stg = smem + OFF_STG + (t * 2 + half) * STG;
        float4 *sY = (float4 *)(smem + OFF_STG + t * 2 * STG);  // [row]: after half 0's columns, then after all
        float4 *sDY = sY + TILE;
        const uint32_t tacc = tmem + (uint32_t)(t * MLP_H + half * 128) + ((uint32_t)((warp & 3) * 32) << 16);
        const float4 *w4 = s_w4 + half * 128;
        uint32_t ngemm = 0;  // accumulators taken so far
        // A written: visible to the tensor cores, the accumulator free
        auto publish = [&]() {
            tc_fence_proxy_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) tc_arrive(&ready[t]);
        };
        auto take = [&]() -> bool {
            // the tile's threads agree, so that none waits for one that gave up
            if (!tc_bar_and(bar_tile, 256, tc_mbar_wait(&done[t], ngemm & 1))) return false;
            ++ngemm;
            tc_fence_after();
            return true;
        };
        // dW4 sums over row quarter `warp & 3`: chunk c, column 16 c + 4 (lane & 3)
        // + (lane >> 3), outputs 2 ((lane >> 2) & 1) and the next
        float2 gw4[8] = {};
        float gb4[MLP_OUT] = {}, loss = 0.f;  // half 0: sums over this thread's rows
        for (int p = 0; p < npairs; ++p) {
            const int tile = ((int)blockIdx.x + p * (int)gridDim.x) * 2 + t;
            const size_t tbase = (size_t)tile * TILE_ELEMS;
            const size_t gr = (size_t)tile * TILE + row;
            // where this thread's 8-column group cg of a tile goes: A and the
            // tiles in global memory (core matrices), gelu' ([cg][row])
            const size_t arow = (size_t)((row >> 3) * (MLP_H / 8) * 64 + (row & 7) * 8) + half * 16 * 64;
            const size_t grow = tbase + (size_t)(half * 16 * TILE + row) * 8;
            // ---- the tile's inputs, in the staging (128 rows of 8) ----
            float *sX = (float *)sY;
            const int tt = tid & 255;
            *(float4 *)(sX + tt * 4) = load_row4(a.X + (size_t)tile * TILE * MLP_XS + tt * 4, a.aligned);
            const float4 tg = load_row4(a.T + gr * MLP_OUT, a.aligned), wt = load_row4(a.w + gr * MLP_OUT, a.aligned);
            tc_bar_sync(bar_tile, 256);
            // ---- as exact sums of three bf16 pieces, and a one (the bias): the
            // operand of the input layer's gradient ----
            if (half == 0) {
                float x[MLP_IN], p0[8], p1[8], p2[8];
                lds8(x, sX + row * MLP_XS);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    p0[i] = bf2f(f2bf(x[i]));
                    p1[i] = bf2f(f2bf(x[i] - p0[i]));
                    p2[i] = x[i] - p0[i] - p1[i];
                }
                uint16_t *xp = a.b.Xp + (size_t)tile * TILE * XP_COLS + (row >> 3) * (XP_COLS / 8) * 64 + (row & 7) * 8;
                *(uint4 *)xp = pack8(p0);
                *(uint4 *)(xp + 64) = pack8(p1);
                *(uint4 *)(xp + 128) = pack8(p2);
                *(uint4 *)(xp + 192) = make_uint4(0x3F80u, 0u, 0u, 0u);
            }
            // ---- input layer: thread = four columns (their weights in registers)
            // of every eighth row, twice ----
#pragma unroll 1
            for (int s = 0; s < 2; ++s) {
                // lanes: two halves of an 8-column group, 8 rows, two groups
                const int cg = (warp & 7) * 4 + s * 2 + (lane >> 4), hc = lane & 1, r0 = (lane >> 1) & 7;
                const int f = cg * 8 + hc * 4;
                float2 w[MLP_IN][2], bz[2];
                {
                    const float4 b = *(const float4 *)(s_bias + f);
                    bz[0] = make_float2(b.x, b.y);
                    bz[1] = make_float2(b.z, b.w);
                }
#pragma unroll
                for (int i = 0; i < MLP_IN; ++i) {
                    const float4 u = __ldg((const float4 *)(a.P + MLP_OFF_W0 + i * MLP_H + f));
                    w[i][0] = make_float2(u.x, u.y);
                    w[i][1] = make_float2(u.z, u.w);
                }
                const float *xr = sX + r0 * MLP_XS;
                const size_t o0 = (size_t)(cg * 64 + r0 * 8 + hc * 4);
                uint16_t *G0 = a.b.G[0] + tbase + (size_t)(cg * TILE + r0) * 8 + hc * 4;
#pragma unroll 2
                for (int k = 0; k < TILE / 8; ++k) {
                    float x[MLP_IN];
                    lds8(x, xr + k * 8 * MLP_XS);
                    uint32_t hv[2], gv[2];
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        float2 z = bz[q];
#pragma unroll
                        for (int i = 0; i < MLP_IN; ++i) z = __ffma2_rn(make_float2(x[i], x[i]), w[i][q], z);
                        float2 h, g;
                        gelu_both(z, h, g);
                        hv[q] = pack_bf16x2(h.x, h.y);
                        gv[q] = pack_bf16x2(g.x, g.y);
                    }
                    const size_t o = o0 + (size_t)k * (MLP_H / 8) * 64;
                    *(uint2 *)(sA + o) = make_uint2(hv[0], hv[1]);
                    *(uint2 *)(a.b.H[0] + tbase + o) = make_uint2(hv[0], hv[1]);
                    *(uint2 *)(G0 + k * 64) = make_uint2(gv[0], gv[1]);
                }
            }
            publish();
            // ---- hidden layers 2 and 3 ----
#pragma unroll 1
            for (int j = 1; j < 3; ++j) {
                if (!(ok = take())) break;
                const float *bias = s_bias + j * MLP_H + half * 128;
                uint16_t *Hj = a.b.H[j] + tbase + arow, *Gj = a.b.G[j] + grow;
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {
                    float v[32];
                    tc_ld32(tacc + (uint32_t)(c * 32), v);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int cg = c * 4 + k;
                        float h[8], g[8];
#pragma unroll
                        for (int q = 0; q < 8; q += 2) {
                            float2 hh, gg;
                            gelu_both(__fadd2_rn(make_float2(v[8 * k + q], v[8 * k + q + 1]),
                                                 *(const float2 *)(bias + cg * 8 + q)),
                                      hh, gg);
                            h[q] = hh.x, h[q + 1] = hh.y, g[q] = gg.x, g[q + 1] = gg.y;
                        }
                        const uint4 hv = pack8(h);
                        *(uint4 *)(sA + arow + cg * 64) = hv;
                        *(uint4 *)(Hj + cg * 64) = hv;
                        *(uint4 *)(Gj + (size_t)cg * TILE * 8) = pack8(g);
                    }
                }
                publish();
            }
            if (!ok || !(ok = take())) break;
            // ---- last hidden layer; the activations replace their accumulator in
            // tensor memory and gelu' goes where A was, for the passes below ----
            {
                const float *bias = s_bias + 3 * MLP_H + half * 128;
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {
                    float v[32];
                    tc_ld32(tacc + (uint32_t)(c * 32), v);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        float g[8];
#pragma unroll
                        for (int q = 0; q < 8; q += 2) {
                            const int cc = 8 * k + q;
                            float2 h, gg;
                            gelu_both(__fadd2_rn(make_float2(v[cc], v[cc + 1]), *(const float2 *)(bias + c * 32 + cc)), h,
                                      gg);
                            v[cc] = h.x, v[cc + 1] = h.y, g[q] = gg.x, g[q + 1] = gg.y;
                        }
                        *(uint4 *)(sA + arow + (c * 4 + k) * 64) = pack8(g);
                    }
                    tc_st16(tacc + (uint32_t)(c * 32), (const uint32_t *)v);
                    tc_st16(tacc + (uint32_t)(c * 32 + 16), (const uint32_t *)(v + 16));
                }
                tc_wait_st();
            }
            // ---- output layer: y = b4 + H4 W4 in the order of the features, the
            // second half's threads going on from the first half's ----
#pragma unroll 1
            for (int hh = 0; hh < 2; ++hh) {
                if (half == hh) {
                    const float4 y = hh == 0 ? __ldg((const float4 *)(a.P + MLP_OFF_B4)) : sY[row];
                    float2 y01 = make_float2(y.x, y.y), y23 = make_float2(y.z, y.w);
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        float v[32];
                        tc_ld32(tacc + (uint32_t)(c * 32), v);
#pragma unroll
                        for (int k = 0; k < 32; ++k) {
                            const float4 wv = w4[c * 32 + k];
                            y01 = __ffma2_rn(make_float2(v[k], v[k]), make_float2(wv.x, wv.y), y01);
                            y23 = __ffma2_rn(make_float2(v[k], v[k]), make_float2(wv.z, wv.w), y23);
                        }
                    }
                    sY[row] = make_float4(y01.x, y01.y, y23.x, y23.y);
                }
                tc_bar_sync(bar_tile, 256);
            }
            float4 d;
            {
                const float4 y = sY[row];
                const float e0 = y.x - tg.x, e1 = y.y - tg.y, e2 = y.z - tg.z, e3 = y.w - tg.w;
                d = make_float4(2.f * wt.x * e0 * a.inv_n, 2.f * wt.y * e1 * a.inv_n, 2.f * wt.z * e2 * a.inv_n,
                                2.f * wt.w * e3 * a.inv_n);
                if (half == 0) {
                    sDY[row] = d;
                    float l = wt.x * e0 * e0;
                    l = fmaf(wt.y * e1, e1, l);
                    l = fmaf(wt.z * e2, e2, l);
                    l = fmaf(wt.w * e3, e3, l);
                    loss += l * a.inv_n;
                    gb4[0] += d.x, gb4[1] += d.y, gb4[2] += d.z, gb4[3] += d.w;
                }
            }
            tc_bar_sync(bar_tile, 256);
            // ---- dW4: sums over rows ----
            // 16 columns of a tile half at a time go through shared memory (16-byte
            // units permuted in each pair of rows: no bank conflicts either way);
            // a thread multiplies 4 rows x 4 columns, the 8 lanes that hold the
            // same columns share out the 16 sums, and these rotate through gw4 so
            // that the loop stays rolled
            {
                const int r0 = (warp & 3) * 32 + (lane >> 2) * 4, cq = lane & 3;
                auto unit = [](int r, int u) {
                    const int line = r >> 1;
                    return line * 128 + ((((r & 1) << 2) | u) ^ ((line & 3) | ((line << 1) & 4))) * 16;
                };
                float4 dd[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) dd[i] = sDY[r0 + i];
                tc_bar_sync(bar_tile, 256);  // the staging takes the place of y and dY
#pragma unroll 1
                for (int c = 0; c < 8; ++c) {
                    float v[16];
                    tc_ld16(tacc + (uint32_t)(c * 16), v);
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        *(float4 *)(stg + unit(row, u)) = make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
                    tc_bar_sync(bar_half, 128);
                    float2 s[8] = {};  // [column][output pair]
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 h = *(const float4 *)(stg + unit(r0 + i, cq));
                        const float hc[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            s[2 * k] = __ffma2_rn(make_float2(hc[k], hc[k]), make_float2(dd[i].x, dd[i].y), s[2 * k]);
                            s[2 * k + 1] =
                                __ffma2_rn(make_float2(hc[k], hc[k]), make_float2(dd[i].z, dd[i].w), s[2 * k + 1]);
                        }
                    }
                    // lane bit 4 takes the upper four, bit 3 two of them, bit 2 one
                    share(s, lane, std::integral_constant<int, 4>());
                    share(s, lane, std::integral_constant<int, 2>());
                    share(s, lane, std::integral_constant<int, 1>());
                    const float2 g = __fadd2_rn(gw4[0], s[0]);
#pragma unroll
                    for (int k = 0; k < 7; ++k) gw4[k] = gw4[k + 1];
                    gw4[7] = g;
                    tc_bar_sync(bar_half, 128);
                }
            }
            // ---- dZ4 = (dY W4^T) gelu' ----
#pragma unroll 2
            for (int cg = 0; cg < 16; ++cg) {
                const uint4 gv = *(const uint4 *)(sA + arow + cg * 64);
                const uint32_t u[4] = {gv.x, gv.y, gv.z, gv.w};
                uint32_t o[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 wa = w4[cg * 8 + 2 * q], wb = w4[cg * 8 + 2 * q + 1];
                    const float da = fmaf(d.x, wa.x, fmaf(d.y, wa.y, fmaf(d.z, wa.z, d.w * wa.w)));
                    const float db = fmaf(d.x, wb.x, fmaf(d.y, wb.y, fmaf(d.z, wb.z, d.w * wb.w)));
                    o[q] = pack_bf16x2(da * __uint_as_float(u[q] << 16), db * __uint_as_float(u[q] & 0xFFFF0000u));
                }
                const uint4 dv = make_uint4(o[0], o[1], o[2], o[3]);
                *(uint4 *)(sA + arow + cg * 64) = dv;
                *(uint4 *)(a.b.D[3] + tbase + arow + cg * 64) = dv;
            }
            publish();
            // ---- back through the hidden layers ----
#pragma unroll 1
            for (int j = 2; j >= 0; --j) {
                const uint4 *G = (const uint4 *)(a.b.G[j] + grow);
                uint4 gq[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) gq[k] = G[k * TILE];  // in flight during the GEMM
                if (!(ok = take())) break;
                uint16_t *Dj = a.b.D[j] + tbase + arow;
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {
                    float v[32];
                    tc_ld32(tacc + (uint32_t)(c * 32), v);
                    uint4 gn[4];
                    if (c < 3) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) gn[k] = G[(c * 4 + 4 + k) * TILE];
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int cg = c * 4 + k;
                        const uint32_t u[4] = {gq[k].x, gq[k].y, gq[k].z, gq[k].w};
                        uint32_t o[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const float2 m = __fmul2_rn(make_float2(v[8 * k + 2 * q], v[8 * k + 2 * q + 1]),
                                                        make_float2(__uint_as_float(u[q] << 16),
                                                                    __uint_as_float(u[q] & 0xFFFF0000u)));
                            o[q] = pack_bf16x2(m.x, m.y);
                        }
                        const uint4 dv = make_uint4(o[0], o[1], o[2], o[3]);
                        if (j > 0) *(uint4 *)(sA + arow + cg * 64) = dv;
                        *(uint4 *)(Dj + cg * 64) = dv;
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) gq[k] = gn[k];
                }
                if (j > 0) publish();
            }
            if (!ok) break;
        }
        // ---- this CTA's sums of dW4, db4 and the loss, in a fixed order ----
        if (!ok) atomicExch(a.err, -9);
        tc_bar_sync(7, 512);
        float *red = (float *)smem;  // [tile][row quarter][half * 128 + column][4], then the row sums
#pragma unroll
        for (int c = 0; c < 8; ++c)
            *(float2 *)(red +
                        ((t * 4 + (warp & 3)) * MLP_H + half * 128 + c * 16 + (lane & 3) * 4 + (lane >> 3)) * 4 +
                        ((lane >> 2) & 1) * 2) = gw4[c];
        float s5[5] = {gb4[0], gb4[1], gb4[2], gb4[3], loss};
#pragma unroll
        for (int k = 0; k < 5; ++k)
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) s5[k] += __shfl_xor_sync(0xffffffffu, s5[k], off);
        float *rs = red + 8 * MLP_H * 4;
        if (half == 0 && lane == 0)
#pragma unroll
            for (int k = 0; k < 5; ++k) rs[(t * 4 + (warp & 3)) * 5 + k] = s5[k];
        tc_bar_sync(7, 512);
        float *po = a.b.part_o + (size_t)blockIdx.x * PB_O;
        for (int i = tid; i < MLP_H * MLP_OUT; i += 512) {
            float s = 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) s += red[k * MLP_H * 4 + i];
            po[i] = s;
        }
        if (tid < 5) {
            float s = 0.f;
            for (int k = 0; k < 8; ++k) s += rs[k * 5 + tid];
            po[MLP_H * MLP_OUT + tid] = s;
        }
    }
    // (after a wait that ran out, the MMAs still in flight get a bounded wait too)
    if (warp == 16 && !ok) {
        if (lane == 0) atomicExch(a.err, -9);
        __syncwarp();
        tc_commit_warp(&drain);
        tc_mbar_wait(&drain, 0);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 16) tc_tmem_free(tmem, 2 * MLP_H);
}

// ---------------------------------------------------------------------------
// weight gradients
// ---------------------------------------------------------------------------
// Job j = 1..3: dWt_j = dZ_{j+1}^T H_j and db_j; j = 0: the input layer, with
// the input pieces (and their column of ones for db0) as the B operand.  A
// stage is 64 samples: 32 KB of dZ and 32 KB of H (4 KB of pieces).
const int GS = 64;
const int GSTAGES = 3;
const uint32_t GA_BYTES = GS * MLP_H * 2, GB_BYTES = GS * MLP_H * 2, GX_BYTES = GS * XP_COLS * 2;
const int GRAD_THREADS = 288;
const int GRAD_SMEM = GSTAGES * (int)(GA_BYTES + GB_BYTES);

struct GradArgs {
    MlpTrainBuf b;
    int units;              // stages of 64 samples in the batch
    int splits[4];          // CTAs of each job
    int cta0[4];            // its first CTA
    size_t off[4];          // its partials in part_w
    int *err;
};

// MN-major variant of the instruction descriptor: both operands transposed
__device__ __forceinline__ uint32_t idesc_mn(int M, int N)
{
    return tc_idesc_bf16(M, N) | (1u << 15) | (1u << 16);
}

__global__ void __launch_bounds__(GRAD_THREADS, 1) mlp_grad_kernel(const GradArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t full[GSTAGES], empty[GSTAGES], done;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int j = 0;
    while (j < 3 && (int)blockIdx.x >= a.cta0[j + 1]) ++j;
    const int s = (int)blockIdx.x - a.cta0[j], S = a.splits[j];
    const int u0 = (int)((int64_t)a.units * s / S), u1 = (int)((int64_t)a.units * (s + 1) / S);
    const bool bias = j > 0;  // the column sums of dZ by warps 0..7
    if (warp == 8) tc_tmem_alloc(&tmem_slot, 512);
    if (tid == 0) {
        for (int i = 0; i < GSTAGES; ++i) {
            tc_mbar_init(&full[i], 1);
            tc_mbar_init(&empty[i], bias ? 9 : 1);
        }
        tc_mbar_init(&done, 1);
        tc_fence_init();
        s_fail = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int n = u1 - u0;
    float acc[8] = {};
    if (warp == 8) {
        const int N = j > 0 ? MLP_H : XP_COLS;
        const uint32_t bbytes = j > 0 ? GB_BYTES : GX_BYTES, bgroup = (uint32_t)(N / 8) * 128;
        const unsigned char *A = (const unsigned char *)a.b.D[j] + (size_t)u0 * GA_BYTES;
        const unsigned char *B =
            (j > 0 ? (const unsigned char *)a.b.H[j - 1] : (const unsigned char *)a.b.Xp) + (size_t)u0 * bbytes;
        const uint32_t idesc = idesc_mn(128, N);
        auto load = [&](int i) {
            const int st = i % GSTAGES;
            unsigned char *d = smem + st * (GA_BYTES + GB_BYTES);
            tc_load_warp(d, A + (size_t)i * GA_BYTES, GA_BYTES, GA_BYTES + bbytes, &full[st]);
            tc_load_warp(d + GA_BYTES, B + (size_t)i * bbytes, bbytes, 0, &full[st]);
        };
        int loaded = 0, i = 0;
        for (; loaded < n && loaded < GSTAGES; ++loaded) load(loaded);
        bool ok = true;
#pragma unroll 1
        for (; i < n; ++i) {
            const int st = i % GSTAGES;
            if (!(ok = tc_mbar_wait(&full[st], (uint32_t)(i / GSTAGES) & 1))) break;
            tc_fence_after();
            const uint32_t a0 = tc_smem(smem + st * (GA_BYTES + GB_BYTES));
            // MN-major, no swizzle: 8-feature groups 128 bytes apart (the
            // stride offset), 8-sample groups one row of core matrices apart
            // (the leading offset)
            const uint64_t da = tc_desc(a0, 4096, 128), db = tc_desc(a0 + GA_BYTES, bgroup, 128);
#pragma unroll
            for (int ks = 0; ks < GS / 16; ++ks)
#pragma unroll
                for (int m = 0; m < 2; ++m)
                    tc_mma_warp(tmem + (uint32_t)(m * 256), da + (uint64_t)((m * 2048 + ks * 8192) >> 4),
                                db + (uint64_t)((ks * 2 * bgroup) >> 4), idesc, (i > 0 || ks > 0) ? 1u : 0u);
            tc_commit_warp(&empty[st]);
            if (i > 0 && loaded < n) {
                const int p = i - 1;
                if (!(ok = tc_mbar_wait(&empty[p % GSTAGES], (uint32_t)(p / GSTAGES) & 1))) break;
                load(loaded++);
            }
        }
        tc_commit_warp(&done);
        if (!ok) {
            s_fail = 1;
            for (int k = i; k < loaded; ++k) tc_mbar_wait(&full[k % GSTAGES], (uint32_t)(k / GSTAGES) & 1);
        }
    } else if (bias) {
        // thread: 8 features (group lane) x 8 samples (group warp) of a stage,
        // the samples in an order that keeps the lanes on different banks
        bool ok = true;
        for (int i = 0; i < n && ok; ++i) {
            const int st = i % GSTAGES;
            ok = tc_mbar_wait(&full[st], (uint32_t)(i / GSTAGES) & 1);
            if (!ok) break;
            const unsigned char *p = smem + st * (GA_BYTES + GB_BYTES) + warp * 4096 + lane * 128;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const uint4 q = *(const uint4 *)(p + ((r + lane) & 7) * 16);
                const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    acc[2 * k] += __uint_as_float(u[k] << 16);
                    acc[2 * k + 1] += __uint_as_float(u[k] & 0xFFFF0000u);
                }
            }
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem(&empty[st])) : "memory");
        }
        if (!ok) s_fail = 1;
    }
    bool ok = tc_mbar_wait(&done, 0);
    if (__syncthreads_or(!ok || s_fail)) {
        if (tid == 0) atomicExch(a.err, -9);
    } else {
        tc_fence_after();
        float *part = a.b.part_w + a.off[j] + (size_t)s * (j > 0 ? PB_H : PB_0);
        const int f = ((warp >> 2) & 1) * 128 + (warp & 3) * 32 + lane;  // output feature
        if (warp < 8) {
            const uint32_t ta = tmem + (uint32_t)((warp >> 2) * 256) + ((uint32_t)((warp & 3) * 32) << 16);
            if (j > 0) {
#pragma unroll 1
                for (int c = 0; c < 8; ++c) {
                    float v[32];
                    if (n > 0)
                        tc_ld32(ta + (uint32_t)(c * 32), v);
                    else
#pragma unroll
                        for (int k = 0; k < 32; ++k) v[k] = 0.f;
                    float4 *o = (float4 *)(part + (size_t)f * MLP_H + c * 32);
#pragma unroll
                    for (int k = 0; k < 8; ++k) o[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
                }
            } else {
                float v[32];
                if (n > 0)
                    tc_ld32(ta, v);
                else
#pragma unroll
                    for (int k = 0; k < 32; ++k) v[k] = 0.f;
#pragma unroll
                for (int i = 0; i < MLP_IN; ++i) part[i * MLP_H + f] = v[i] + (v[8 + i] + v[16 + i]);
                part[MLP_IN * MLP_H + f] = v[24];
            }
        }
        if (bias) {
            // column sums: the 8 sample groups in a fixed order; feature 8 lane + k
            float *red = (float *)smem;
            if (warp < 8)
#pragma unroll
                for (int k = 0; k < 8; ++k) red[(warp * 8 + k) * 32 + lane] = acc[k];
            __syncthreads();
            if (tid < MLP_H) {
                float sum = 0.f;
#pragma unroll
                for (int g = 0; g < 8; ++g) sum += red[(g * 8 + (tid & 7)) * 32 + (tid >> 3)];
                part[MLP_H * MLP_H + tid] = sum;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) tc_tmem_free(tmem, 512);
}

// ---------------------------------------------------------------------------
// update
// ---------------------------------------------------------------------------
__device__ __forceinline__ void write_blocks(const MlpBlocks &k, int j, int e, float w)
{
    const int out = e >> 8, in = e & 255;
    const uint16_t b = f2bf(w);
    k.Wf[j][mlp_chunk_index(out, in)] = b;
    k.Wb[j][mlp_chunk_index(in, out)] = b;
    k.Wt[j][tc_core_offset(out, in, MLP_H) / 2] = b;
    const int q = (out >> 7) * 2 + (in >> 7);
    // halved (exact in BF16): the serving kernel's GELU takes z / 2
    k.Wq[j][(size_t)q * 128 * 128 + tc_core_offset(out & 127, in & 127, 128) / 2] = f2bf(0.5f * w);
}

// hidden layer (1..3) and element of its weight matrix of parameter i, or 0
__device__ __forceinline__ int hidden_element(int i, int &e)
{
    const int k = i - MLP_OFF_WT(1);
    if (k < 0 || i >= MLP_OFF_W4) return 0;
    const int j = k / PB_H;
    e = k - j * PB_H;
    return e < MLP_H * MLP_H ? j + 1 : 0;
}

struct UpdateArgs {
    const float *part_w, *part_o;
    int splits[4];
    size_t off[4];
    int no;  // partials of the output layer
    const int *err;
    MlpAdam m;
    MlpBlocks blk;
};

// one thread per parameter (and one for the loss).  After a wait that ran out,
// in this step or before it, the partial sums are incomplete: nothing changes.
__global__ void __launch_bounds__(256) mlp_update_kernel(const UpdateArgs a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > MLP_NPARAM || *a.err != 0) return;
    const float *p;
    int cnt, stride;
    if (i >= MLP_OFF_W4) {
        p = a.part_o + (i - MLP_OFF_W4);
        cnt = a.no;
        stride = PB_O;
    } else if (i < MLP_OFF_WT(1)) {
        p = a.part_w + a.off[0] + i;
        cnt = a.splits[0];
        stride = PB_0;
    } else {
        const int k = i - MLP_OFF_WT(1), j = k / PB_H;
        p = a.part_w + a.off[j + 1] + (k - j * PB_H);
        cnt = a.splits[j + 1];
        stride = PB_H;
    }
    float g0 = 0.f, g1 = 0.f, g2 = 0.f, g3 = 0.f;
    int s = 0;
    for (; s + 8 <= cnt; s += 8) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = __ldcs(p + (size_t)(s + k) * stride);
        g0 += v[0] + v[4];
        g1 += v[1] + v[5];
        g2 += v[2] + v[6];
        g3 += v[3] + v[7];
    }
    for (; s < cnt; ++s) g0 += __ldcs(p + (size_t)s * stride);
    const float g = (g0 + g1) + (g2 + g3);
    if (i == MLP_NPARAM) {
        *a.m.loss = g;
        return;
    }
    a.m.G[i] = g;
    if (a.m.lr == 0.f) return;
    const float mi = a.m.b1 * a.m.m[i] + (1.f - a.m.b1) * g;
    const float vi = a.m.b2 * a.m.v[i] + (1.f - a.m.b2) * g * g;
    a.m.m[i] = mi;
    a.m.v[i] = vi;
    const float w = a.m.P[i] - a.m.lr * (mi * a.m.c1) / (sqrtf(vi * a.m.c2) + a.m.eps);
    a.m.P[i] = w;
    int e;
    const int j = hidden_element(i, e);
    if (j > 0) write_blocks(a.blk, j - 1, e, w);
}

__global__ void __launch_bounds__(256) mlp_blocks_kernel(const float *__restrict__ P, MlpBlocks k)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= MLP_NPARAM) return;
    int e;
    const int j = hidden_element(i, e);
    if (j > 0) write_blocks(k, j - 1, e, P[i]);
}

// CTAs of the weight-gradient jobs: one per SM in all, shared out by the bytes
// a job reads (the input layer's pieces are an eighth of an activation tile)
void grad_splits(int units, int nsm, int *splits)
{
    int s0 = (int)(0.15 * nsm), sh = (nsm - s0) / 3;
    s0 = std::max(1, std::min(s0, units));
    sh = std::max(1, std::min(sh, units));
    splits[0] = s0;
    for (int j = 1; j < 4; ++j) splits[j] = sh;
}

// CTAs of the step kernel: one per SM, each with pairs of tiles
int step_grid(int pairs, int nsm) { return std::max(1, std::min(pairs, nsm)); }

}  // namespace

size_t mlp_train_part_w(int batch, int nsm)
{
    int s[4];
    grad_splits(std::max(batch / GS, 1), nsm, s);
    return (size_t)s[0] * PB_0 + (size_t)(s[1] + s[2] + s[3]) * PB_H;
}

size_t mlp_train_part_o(int batch, int nsm)
{
    return (size_t)step_grid(batch / (2 * TILE), nsm) * PB_O;
}

cudaError_t launch_mlp_blocks(const float *P, const MlpBlocks &blk, cudaStream_t st)
{
    mlp_blocks_kernel<<<(MLP_NPARAM + 255) / 256, 256, 0, st>>>(P, blk);
    return cudaGetLastError();
}

cudaError_t launch_mlp_train(const float *X, const float *T, const float *w, int n, const MlpTrainBuf &buf,
                             const MlpBlocks &blk, const MlpAdam &adam, int *err, int nsm, cudaStream_t st)
{
    StepArgs a;
    a.X = X;
    a.T = T;
    a.w = w;
    a.P = adam.P;
    for (int j = 0; j < 3; ++j) {
        a.Wf[j] = blk.Wf[j];
        a.Wb[j] = blk.Wb[j];
    }
    a.b = buf;
    a.pairs = n / (2 * TILE);
    a.aligned = ((((uintptr_t)X) | ((uintptr_t)T) | ((uintptr_t)w)) & 15) == 0;
    a.inv_n = 1.0f / n;
    a.err = err;
    const int grid = step_grid(a.pairs, nsm);
    static std::atomic<uint64_t> step_attr{0}, grad_attr{0};
    cudaError_t e = set_dynamic_smem(step_attr, mlp_step_kernel, STEP_SMEM);
    if (e == cudaSuccess) e = set_dynamic_smem(grad_attr, mlp_grad_kernel, GRAD_SMEM);
    if (e != cudaSuccess) return e;
    mlp_step_kernel<<<grid, STEP_THREADS, STEP_SMEM, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    GradArgs ga;
    ga.b = buf;
    ga.units = n / GS;
    grad_splits(ga.units, nsm, ga.splits);
    size_t off = 0;
    int cta = 0;
    for (int j = 0; j < 4; ++j) {
        ga.cta0[j] = cta;
        ga.off[j] = off;
        cta += ga.splits[j];
        off += (size_t)ga.splits[j] * (j > 0 ? PB_H : PB_0);
    }
    ga.err = err;
    mlp_grad_kernel<<<cta, GRAD_THREADS, GRAD_SMEM, st>>>(ga);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    UpdateArgs ua;
    ua.part_w = buf.part_w;
    ua.part_o = buf.part_o;
    for (int j = 0; j < 4; ++j) {
        ua.splits[j] = ga.splits[j];
        ua.off[j] = ga.off[j];
    }
    ua.no = grid;
    ua.err = err;
    ua.m = adam;
    ua.blk = blk;
    mlp_update_kernel<<<(MLP_NPARAM + 256) / 256, 256, 0, st>>>(ua);
    return cudaGetLastError();
}
