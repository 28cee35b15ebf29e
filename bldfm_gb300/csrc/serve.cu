// Serving path of the learned surrogate (footprint mode, MOST profiles): the
// per-mode sweep of the FP32 solver is replaced by the MLP's transfer at z_m.
// One thread per solved mode in each kernel; the spectra kernel writes the
// same (Xp, Xq) slots and Hermitian mirrors as the sweep, so the output
// transform is the solver's own.
#include "devattr.h"
#include "../../include/bldfm_gb300.h"
#include "devmath.cuh"
#include "mlp_common.cuh"
#include "serve.h"
#include "surrogate_phys.cuh"
#include "tc.cuh"

#include <algorithm>

namespace {

// rotated, scaled wavenumbers of mode m: k_par (signed), |k_perp|, |k|
__device__ __forceinline__ void mode_k(const SolveGeom &g, uint32_t e, float ax, float ay, float zm, int &r, int &c,
                                       bool &paired, float &kpar, float &kperp, float &k)
{
    unpack_mode(e, r, c, paired);
    const float lx = ax * (float)freq_of_index(c, g.nlx), ly = ay * (float)freq_of_index(r, g.nly);
    kpar = zm * fmaf(g.ex, lx, g.ey * ly);
    kperp = fabsf(zm * fmaf(-g.ey, lx, g.ex * ly));
    k = sqrtf(fmaf(kpar, kpar, kperp * kperp));
}

__global__ void sur_features_kernel(const SolveGeom g, const uint32_t *__restrict__ modes, float ax, float ay,
                                    float zm, float s1, float s2, float s3, float *__restrict__ X, int64_t npad)
{
    const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= npad) return;
    float kpar = 1.f, kperp = 0.f;
    if (m < g.nsolved) {
        int r, c;
        bool paired;
        float k;
        mode_k(g, modes[m], ax, ay, zm, r, c, paired, kpar, kperp, k);
        kpar = fabsf(kpar);
    }
    feature_row(X + (size_t)m * 8, kpar, kperp, s1, s2, s3);
}

__global__ void sur_exact_kernel(const SolveGeom g, const uint32_t *__restrict__ modes, float ax, float ay, float zm,
                                 const TransferCase *__restrict__ tc, const float4 *__restrict__ steps,
                                 float *__restrict__ Y)
{
    const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= g.nsolved) return;
    int r, c;
    bool paired;
    float kpar, kperp, k;
    mode_k(g, modes[m], ax, ay, zm, r, c, paired, kpar, kperp, k);
    transfer_one(*tc, steps, fabsf(kpar), kperp, Y + (size_t)m * 4);
}

// (Xp, Xq) of solved mode e and its Hermitian mirror from the targets y
__device__ __forceinline__ void emit_spectrum(const SolveGeom &g, uint32_t e, const float *y, float ax, float ay,
                                              float zm, float inv_wind, float ktop, float utop,
                                              float2 *__restrict__ Xp, float2 *__restrict__ Xq)
{
    int r, c;
    bool paired;
    float kpar, kperp, k;
    mode_k(g, e, ax, ay, zm, r, c, paired, kpar, kperp, k);
    float2 Tq, Rt;
    decode_transfer(y, k, Tq, Rt);
    Rt = sp_cmul(Rt, top_ratio(ktop, utop, fabsf(kpar), kperp));
    if (kpar < 0.f) {
        Tq.y = -Tq.y;
        Rt.y = -Rt.y;
    }
    const float q0 = g.q0dc_f;
    float2 q = make_float2(q0 * Tq.x, q0 * Tq.y);
    float2 p = sp_cmul(make_float2(Rt.x * inv_wind, Rt.y * inv_wind), q);
    if (g.do_shift) {
        const int kx = freq_of_index(c, g.nlx), ky = freq_of_index(r, g.nly);
        const uint32_t turns = (uint32_t)kx * g.turn_x + (uint32_t)ky * g.turn_y;
        float sn, cs;
        sincospif((float)(int32_t)turns * 4.656612873077393e-10f, &sn, &cs);
        const float2 sh = make_float2(cs, sn);
        p = sp_cmul(p, sh);
        q = sp_cmul(q, sh);
    }
    Xp[spec_idx(g, 0, r, c)] = p;
    Xq[spec_idx(g, 0, r, c)] = q;
    if (paired) {
        const int rm = index_of_freq(-freq_of_index(r, g.nly), g.nly);
        const int cm = index_of_freq(-freq_of_index(c, g.nlx), g.nlx);
        Xp[spec_idx(g, 0, rm, cm)] = make_float2(p.x, -p.y);
        Xq[spec_idx(g, 0, rm, cm)] = make_float2(q.x, -q.y);
    }
}

__global__ void sur_spectra_kernel(const SolveGeom g, const uint32_t *__restrict__ modes, const float *__restrict__ Y,
                                   float ax, float ay, float zm, float inv_wind, float ktop, float utop,
                                   float2 *__restrict__ Xp, float2 *__restrict__ Xq)
{
    const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= g.nsolved) return;
    emit_spectrum(g, modes[m], Y + (size_t)m * 4, ax, ay, zm, inv_wind, ktop, utop, Xp, Xq);
}

// ---------------------------------------------------------------------------
// Fused serving kernel (sur_serve_kernel) and its helpers
// ---------------------------------------------------------------------------
#define SV_K0 32     // K of the split input layer
#define SV_WARPS 16  // epilogue warps: 4 per TMEM lane quarter, each 2 x 16 columns of a half
#define SV_OUT_GROUPS 2  // column groups of the output layer's partial sums
#define SV_ROWS 64  // threads of the two row warps (features, spectra), two rows each
// + one control warp (copies and MMAs): 19 warps, five a scheduler, which would
// leave 96 registers a thread.  At 88 two warps of the exact low band's kernel
// fit beside them on every SM (16 footprints of 512^2: network 861 us and band
// 115 after it; 890 with the band, 695, inside).
#define SV_THREADS (32 * SV_WARPS + 32 + SV_ROWS)
#define SV_REGS 88
#define SV_AB(i) (256u + 64u * (uint32_t)(i))  // TMEM column of activation K-half buffer i

struct SvSmem {
    uint16_t Wq[4][128 * 128];   // Wt_j quarters (N half, K half), B operands
    uint16_t A0[128 * SV_K0];    // input-layer A operand (split features)
    uint16_t B0[MLP_H * SV_K0];  // split W0 (B operand of the input layer)
    float bias[4][MLP_H];
    float W4[MLP_H * MLP_OUT];
    float4 Yp[2][SV_OUT_GROUPS][128];  // output-layer partial sums, of even and odd tiles
    float b4[4];
};

// Quarter q = 2 nh + kh of Wt_j (Wq_j: four contiguous 32 KB quarters in the
// layout of a 128 x 128 operand) into shared memory: one bulk copy.  Called by
// the whole control warp, as the MMAs are.
__device__ __forceinline__ void sv_load_quarter(uint16_t *dst, const uint16_t *Wq, int q, uint64_t *bar)
{
    const uint32_t bytes = 128 * 128 * 2;
    tc_load_warp(dst, (const char *)Wq + (size_t)q * bytes, bytes, bytes, bar);
}

// D[dcol .. +127] (+)= A[TMEM acol .. +63] (K = 128) x quarter^T: 8 MMAs of
// K = 16; bdesc is the quarter's descriptor (each K step advances the start
// address by 256 bytes, 16 in the descriptor's address field)
__device__ __forceinline__ void sv_mma_quarter(uint32_t dt, uint32_t at, uint64_t bdesc, uint32_t idesc,
                                               bool accumulate)
{
    tc_mma_ts_warp(dt, at, bdesc, idesc, accumulate ? 1u : 0u);
#pragma unroll
    for (int s = 1; s < 8; ++s) tc_mma_ts_warp(dt, at + 8 * s, bdesc + (uint64_t)(16 * s), idesc, 1u);
}

// K steps s0 .. s0 + 3 of a quarter MMA (K = 64 of the 128)
__device__ __forceinline__ void sv_mma_quarter_part(uint32_t dt, uint32_t at, uint64_t bdesc, uint32_t idesc, int s0)
{
#pragma unroll
    for (int s = 0; s < 4; ++s)
        tc_mma_ts_warp(dt, at + 8 * (s0 + s), bdesc + (uint64_t)(16 * (s0 + s)), idesc, 1u);
}

// Bounded wait of a whole converged warp for phase `parity` of an mbarrier
// that also gives up as soon as another warp has recorded a failure in *fail.
// The wait suspends: warps that poll take the issue slots of the ones that
// compute (1374 us for the kernel where suspended waits take 938).
__device__ __forceinline__ bool sv_wait(uint64_t *bar, uint32_t parity, const volatile int *fail)
{
    const uint32_t a = tc_smem(bar);
    for (long it = 0; it < BLDFM_WAIT_POLLS; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
        if ((it & 63) == 63 && *fail) return false;
    }
    return false;
}

__device__ __forceinline__ void sv_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(tc_smem(bar)) : "memory");
}

// barrier of the row warps; true if all of them pass true
__device__ __forceinline__ bool sv_row_sync(bool ok) { return tc_bar_and(2, SV_ROWS, ok); }

// true for a mode that the exact low band writes (lowband_mode's enumeration
// and its disc, operation for operation)
__device__ __forceinline__ bool sv_in_band(const SurCase &c, uint32_t e)
{
    int r, col;
    bool paired;
    unpack_mode(e, r, col, paired);
    const int kx = freq_of_index(col, c.g.nlx), ky = freq_of_index(r, c.g.nly);
    const float lx = c.ax * (float)kx, ly = c.ay * (float)ky;
    return abs(kx) <= c.band_bx && abs(ky) <= c.band_by && fmaf(lx, lx, ly * ly) < c.band_kmax2;
}

// mode word of row r of a tile (0 past the case's last mode)
__device__ __forceinline__ uint32_t sv_mode_word(const SurCase &c, int64_t tile, int r)
{
    const int64_t m = (tile - c.tile0) * 128 + r;
    return m < c.g.nsolved ? c.modes[m] : 0u;
}

// features of row r of a tile (mode word e) -> [xh | xl | xh | 0] (input-layer
// A operand, K = 32)
__device__ __forceinline__ void sv_features(const SurCase &c, int64_t tile, int r, uint32_t e, uint16_t *A0)
{
    const int64_t m = (tile - c.tile0) * 128 + r;
    float kpar = 1.f, kperp = 0.f;
    if (m < c.g.nsolved) {
        int rr, cc;
        bool pr;
        float k;
        mode_k(c.g, e, c.ax, c.ay, c.zm, rr, cc, pr, kpar, kperp, k);
        kpar = fabsf(kpar);
    }
    float x[8], xl[8];
    feature_row(x, kpar, kperp, c.s1, c.s2, c.s3);
#pragma unroll
    for (int i = 0; i < 8; ++i) xl[i] = x[i] - bf2f(f2bf(x[i]));
    const uint4 hi = make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]),
                                pack_bf16x2(x[6], x[7]));
    const uint4 lo = make_uint4(pack_bf16x2(xl[0], xl[1]), pack_bf16x2(xl[2], xl[3]), pack_bf16x2(xl[4], xl[5]),
                                pack_bf16x2(xl[6], xl[7]));
    *(uint4 *)(A0 + tc_core_offset(r, 0, SV_K0) / 2) = hi;
    *(uint4 *)(A0 + tc_core_offset(r, 8, SV_K0) / 2) = lo;
    *(uint4 *)(A0 + tc_core_offset(r, 16, SV_K0) / 2) = hi;
    *(uint4 *)(A0 + tc_core_offset(r, 24, SV_K0) / 2) = make_uint4(0u, 0u, 0u, 0u);
}

// hidden-layer epilogue of 16 columns of this thread's row (FP32 bits r):
// bias, GELU in f32x2 lanes, BF16 pairs into 8 activation columns at ta
__device__ __forceinline__ void sv_epilogue_hidden(const uint32_t *r, uint32_t ta, const float *bias)
{
    uint32_t w[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        const float2 g = gelu2_half(make_float2(__uint_as_float(r[2 * p]), __uint_as_float(r[2 * p + 1])),
                                    *(const float2 *)(bias + 2 * p));
        w[p] = pack_bf16x2(g.x, g.y);
    }
    tc_st8(ta, w);
}

// last hidden layer's epilogue of 32 columns: v <- gelu(v + b)
__device__ __forceinline__ void sv_gelu32(float *v, const float *bias)
{
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        const float2 h = gelu2_half(make_float2(v[i], v[i + 1]), *(const float2 *)&bias[i]);
        v[i] = h.x;
        v[i + 1] = h.y;
    }
}

// ... and its part of the 256 -> 4 output layer: y += v . W4 rows
__device__ __forceinline__ void sv_out32(const float *v, const float4 *w, const float *W4, float4 &y)
{
    // w: the first 4 columns' weights, read before the wait for y; each
    // further 4 are read one group ahead of the chain
    float2 y01 = make_float2(y.x, y.y), y23 = make_float2(y.z, y.w);
    float4 wa[4], wb[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) wa[i] = w[i];
#pragma unroll
    for (int g = 0; g < 8; ++g) {
        if (g < 7)
#pragma unroll
            for (int i = 0; i < 4; ++i) wb[i] = *(const float4 *)&W4[(4 * (g + 1) + i) * MLP_OUT];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float h = v[4 * g + i];
            y01 = __ffma2_rn(make_float2(h, h), make_float2(wa[i].x, wa[i].y), y01);
            y23 = __ffma2_rn(make_float2(h, h), make_float2(wa[i].z, wa[i].w), y23);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) wa[i] = wb[i];
    }
    y = make_float4(y01.x, y01.y, y23.x, y23.y);
}

// Fused serving kernel: features -> MLP -> spectra for 128 modes per tile,
// one persistent CTA per SM: 16 epilogue warps, one control warp and two row
// warps.
//
// All four matrix layers run on the tensor cores (tcgen05.mma, M = 128, FP32
// accumulators in TMEM); the epilogues (bias + GELU) and the 256 -> 4 output
// layer run on the CUDA cores in FP32.  Input layer in BF16 at FP32 accuracy:
// x = xh + xl and W0 = wh + wl split into BF16 parts, K = 32 columns
// [xh | xl | xh | 0] x [wh | wh | wl | 0] give x.W0 up to the xl.wl term
// (relative 2^-16).
//
// Overlap of tensor cores and epilogues: every layer's 256 outputs are two
// N = 128 halves with their own accumulator (TMEM columns 0 and 128) and
// completion barrier.  The epilogue of half 0 writes the low K half of the
// next layer's activations (BF16 pairs in TMEM: the A operand of the next
// MMAs) while the tensor cores finish half 1; the next layer's first quarter
// MMA (half 0, low K) then runs during the epilogue of half 1.  Activations
// rotate through three K-half TMEM buffers so that no buffer is rewritten
// while an MMA reads it.  The hidden weights stream through shared memory as
// four 32 KB quarters (N half x K half), each reloaded with the next layer's
// as soon as the MMAs reading it have completed.  The control warp issues
// every copy and MMA, converged (one elected lane: from a one-lane branch the
// issue took longer than the MMAs), and hands work to the epilogue warps
// through mbarriers only, so a blocked MMA issue never holds an epilogue back.
// The row warps compute the next tile's features and write the last one's
// spectra beside the layers.
//
// What bounds it, in clocks of a tile's 15,300 (16 footprints of 512^2, 109
// tiles an SM, 861 us alone with 96 registers; 1003 with 8 epilogue warps,
// features and spectra on four of them and the MMAs issued from one lane): eight epilogues of a half,
// 1,330 each, where tanh.approx takes 1,088 and the FP32 register ports some
// 1,000; a bubble of 500 to 600 per layer from the end of the half-1 epilogue
// until the last four MMAs of half 0 have completed; and the output layer,
// whose weights come through the shared-memory port (4,096 clocks).  A second
// tile in flight would hide the bubbles, but its activations do not fit TMEM:
// through shared memory the port is the bound (1,034 us).
//
// Every wait is bounded; on a timeout the kernel records BLDFM_ERR_TIMEOUT, all
// warps leave their loops, the control warp waits (bounded) for its copies and
// MMAs in flight, and TMEM is freed.
__global__ void __maxnreg__(SV_REGS)
    sur_serve_kernel(const SurCase *__restrict__ cases, int ncases, int64_t ntiles, const MlpServing net, int *err)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    SvSmem &S = *reinterpret_cast<SvSmem *>(smem_raw);
    // bar_m[h]: MMAs of accumulator half h done; bar_e[h]: epilogue of half h
    // done (one arrival per epilogue warp); bar_f: input operand written (one
    // arrival per row thread); bar_q[q]: weight quarter q loaded
    // bar_p: the first 64 columns of half 1 done (one arrival per epilogue warp)
    // bar_a: the input layer's MMAs have read their operand; bar_x[s]: step s of
    // the output layer's chains of sums done, bar_y[b]: the last step, of an even
    // / odd tile (8 warps each), bar_yf[b]: those sums read (one arrival per row thread)
    __shared__ uint64_t bar_m[2], bar_e[2], bar_p, bar_f, bar_a, bar_x[3], bar_y[2], bar_yf[2], bar_q[4];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    __shared__ SurCase sc[2];         // cases of the current and the next tile (row warps)
    __shared__ int64_t s_case_t1[2];  // first tile after each
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const volatile int *fail = &s_fail;
    if (warp == 0) tc_tmem_alloc(&tmem_slot, 512);
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            tc_mbar_init(&bar_m[i], 1);
            tc_mbar_init(&bar_e[i], SV_WARPS);
            tc_mbar_init(&bar_y[i], 4 * SV_OUT_GROUPS);
            tc_mbar_init(&bar_yf[i], SV_ROWS);
        }
        tc_mbar_init(&bar_f, SV_ROWS);
        tc_mbar_init(&bar_a, 1);
        for (int i = 0; i < 3; ++i) tc_mbar_init(&bar_x[i], 4 * SV_OUT_GROUPS);
        tc_mbar_init(&bar_p, SV_WARPS);
        for (int i = 0; i < 4; ++i) tc_mbar_init(&bar_q[i], 1);
        tc_fence_init();
        s_fail = 0;
    }
    // split W0 / 2 [in][out] into the B operand [out][K = 32]; weights and biases
    // of the hidden layers are halved for gelu2_half
    for (int e = tid; e < MLP_H * SV_K0; e += blockDim.x) {
        const int f = e / SV_K0, k = e % SV_K0, grp = k >> 3, i = k & 7;
        const float w = 0.5f * net.P[MLP_OFF_W0 + i * MLP_H + f];
        const uint16_t wh = f2bf(w);
        const uint16_t wl = f2bf(w - bf2f(wh));
        S.B0[tc_core_offset(f, k, SV_K0) / 2] = grp < 2 ? wh : (grp == 2 ? wl : (uint16_t)0);
    }
    for (int i = tid; i < MLP_H; i += blockDim.x) {
        S.bias[0][i] = 0.5f * net.P[MLP_OFF_B0 + i];
#pragma unroll
        for (int j = 1; j <= 3; ++j) S.bias[j][i] = 0.5f * net.P[MLP_OFF_B(j) + i];
    }
    for (int i = tid; i < MLP_H * MLP_OUT; i += blockDim.x) S.W4[i] = net.P[MLP_OFF_W4 + i];
    if (tid < MLP_OUT) S.b4[tid] = net.P[MLP_OFF_B4 + tid];
    tc_fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    // activation K-half buffers of layers 1..3: (lo, hi) = (0, 1), (2, 0), (1, 2)
    auto buf_lo = [](int j) { return j == 0 ? 0 : (j == 1 ? 2 : 1); };
    auto buf_hi = [](int j) { return j == 0 ? 1 : (j == 1 ? 0 : 2); };

    if (warp == SV_WARPS) {
        // ---------------- control warp: copies and MMAs ----------------
        const uint32_t idesc = tc_idesc_bf16(128, 128);
        uint64_t bq[4];  // descriptors of the weight quarters
        for (int q = 0; q < 4; ++q) bq[q] = tc_desc(tc_smem(S.Wq[q]), 128, 2048);
        const uint64_t da0 = tc_desc(tc_smem(S.A0), 128, 512), db0 = tc_desc(tc_smem(S.B0), 128, 512);
        uint32_t ph_m[2] = {0u, 0u}, ph_e[2] = {0u, 0u}, ph_p = 0u, ph_f = 0u, ph_q[4] = {0u, 0u, 0u, 0u};
        bool pend_m[2] = {false, false}, pend_q[4] = {false, false, false, false};
        bool ok = true;
        if ((int64_t)blockIdx.x < ntiles)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                sv_load_quarter(S.Wq[q], net.Wq[0], q, &bar_q[q]);
                pend_q[q] = true;
            }
        for (int64_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
            // input layer, both halves (B0 rows 128 h .. +127 start 8 KB
            // apart); the previous tile's last epilogue has released both
            // accumulator halves (its bar_e phases were waited below)
            ok = sv_wait(&bar_f, ph_f, fail);
            if (!ok) break;
            ph_f ^= 1u;
            tc_fence_after();
            for (int h = 0; h < 2; ++h) {
                tc_mma_warp(tmem + 128u * h, da0, db0 + (uint64_t)(512 * h), idesc, 0u);
                tc_mma_warp(tmem + 128u * h, da0 + 16u, db0 + (uint64_t)(512 * h + 16), idesc, 1u);
                tc_commit_warp(&bar_m[h]);
                pend_m[h] = true;
            }
            tc_commit_warp(&bar_a);
            for (int j = 0; j < 4 && ok; ++j) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (!ok) break;
                    // layer j's half h is complete: the quarters of Wt_j in N
                    // half h are free for the next layer's (after the last
                    // layer, the next tile's first)
                    ok = sv_wait(&bar_m[h], ph_m[h], fail);
                    if (!ok) break;
                    ph_m[h] ^= 1u;
                    pend_m[h] = false;
                    if (j >= 1) {
                        const uint16_t *next =
                            j < 3 ? net.Wq[j] : (tile + gridDim.x < ntiles ? net.Wq[0] : nullptr);
                        if (next)
#pragma unroll
                            for (int q = 2 * h; q < 2 * h + 2; ++q) {
                                sv_load_quarter(S.Wq[q], next, q, &bar_q[q]);
                                pend_q[q] = true;
                            }
                    }
                    const uint32_t alo = tmem + SV_AB(j < 3 ? buf_lo(j) : 0),
                                   ahi = tmem + SV_AB(j < 3 ? buf_hi(j) : 0);
                    if (h == 1 && j < 3) {
                        // the first 64 activations of the high K half: the
                        // first half of quarter 1 (layer j + 1, N half 0)
                        ok = sv_wait(&bar_p, ph_p, fail) && sv_wait(&bar_q[1], ph_q[1], fail);
                        if (!ok) break;
                        ph_p ^= 1u;
                        ph_q[1] ^= 1u;
                        pend_q[1] = false;
                        tc_fence_after();
                        sv_mma_quarter_part(tmem, ahi, bq[1], idesc, 0);
                    }
                    // the epilogue of half h has read the accumulator (and
                    // written the activations it feeds)
                    ok = sv_wait(&bar_e[h], ph_e[h], fail);
                    if (!ok) break;
                    ph_e[h] ^= 1u;
                    if (j == 3) continue;
                    tc_fence_after();
                    if (h == 1) {
                        sv_mma_quarter_part(tmem, ahi, bq[1], idesc, 4);
                        tc_commit_warp(&bar_m[0]);
                        pend_m[0] = true;
                    }
#pragma unroll
                    for (int q = h == 0 ? 0 : 2; q < (h == 0 ? 1 : 4); ++q) {
                        if (!ok) break;
                        ok = sv_wait(&bar_q[q], ph_q[q], fail);
                        if (!ok) break;
                        ph_q[q] ^= 1u;
                        pend_q[q] = false;
                        sv_mma_quarter(tmem + 128u * (q >> 1), (q & 1) ? ahi : alo, bq[q], idesc, (q & 1) != 0);
                        if (q & 1) {
                            tc_commit_warp(&bar_m[q >> 1]);
                            pend_m[q >> 1] = true;
                        }
                    }
                }
            }
        }
        if (!ok) {
            s_fail = 1;
            if (lane == 0) atomicExch(err, BLDFM_ERR_TIMEOUT);
            const int never = 0;  // drain without the early exit on s_fail
            for (int h = 0; h < 2; ++h)
                if (pend_m[h] && sv_wait(&bar_m[h], ph_m[h], &never)) ph_m[h] ^= 1u;
            // MMAs issued after the last commit: one more commit tracks them all
            tc_commit_warp(&bar_m[0]);
            sv_wait(&bar_m[0], ph_m[0], &never);
            for (int q = 0; q < 4; ++q)
                if (pend_q[q]) sv_wait(&bar_q[q], ph_q[q], &never);
        }
    } else if (warp < SV_WARPS) {
        // ---------------- epilogue warps ----------------
        // warp w owns TMEM lanes 32 (w % 4) .. +31 (its rows) and columns
        // 16 cg .. +15 of each 64 columns of an accumulator half (cg = w / 4);
        // in the last hidden layer, columns 32 cg .. +31 of a half.  The output
        // layer keeps two chains of sums per row: columns 32 c .. and 64 + 32 c
        // .. of half 0, then of half 1, handed from warp to warp through Yp, so
        // that all warps share the layer and the order of the sums stays.
        const int qd = warp & 3, cg = warp >> 2, chain = cg & 1, second = cg >> 1;
        const int row = 32 * qd + lane;
        const uint32_t lane_off = (uint32_t)(32 * qd) << 16;
        uint32_t ph_m[2] = {0u, 0u}, ph_x = 0u, ph_yf[2] = {1u, 1u};
        int par = 0;  // parity of the tile's place in this CTA's sequence
        bool ok = true;
        for (int64_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, par ^= 1) {
            for (int j = 0; j < 3 && ok; ++j) {
                // both halves; half 1's accumulators are read while half 0's
                // activations are on their way to TMEM
                uint32_t r[2][32];
                const uint32_t td = tmem + lane_off + 16u * cg;
                auto load = [&](int h) {
                    ok = sv_wait(&bar_m[h], ph_m[h], fail);
                    ph_m[h] ^= 1u;
                    tc_fence_after();
                    if (ok) tc_ld16x2_issue(td + 128u * h, td + 128u * h + 64u, r[h]);
                };
                auto announce = [&](uint64_t *bar) {
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) sv_arrive(bar);
                };
                load(0);
                if (!ok) break;
                tc_wait_ld32(r[0]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float *bias = S.bias[j] + 128 * h + 16 * cg;
                    const uint32_t ta = tmem + lane_off + SV_AB(h == 0 ? buf_lo(j) : buf_hi(j)) + 8u * cg;
                    sv_epilogue_hidden(r[h], ta, bias);
                    if (h == 1) announce(&bar_p);
                    sv_epilogue_hidden(r[h] + 16, ta + 32u, bias + 64);
                    if (h == 0) {
                        load(1);
                        if (!ok) break;
                    }
                    announce(&bar_e[h]);
                    if (h == 0) tc_wait_ld32(r[1]);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (!ok) break;
                ok = sv_wait(&bar_m[h], ph_m[h], fail);
                if (!ok) break;
                ph_m[h] ^= 1u;
                tc_fence_after();
                float v[32];
                tc_ld32(tmem + lane_off + 128u * h + 32u * cg, v);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) sv_arrive(&bar_e[h]);
                sv_gelu32(v, S.bias[3] + 128 * h + 32 * cg);
                const float *w4 = S.W4 + (128 * h + 32 * cg) * MLP_OUT;
                float4 w0[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) w0[i] = *(const float4 *)&w4[i * MLP_OUT];
                // step 2 h + second of the chain: after the one before, the
                // first when the sums of the tile before last have been read
                float4 &Yp = S.Yp[par][chain][row];
                float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
                if (h == 0 && second == 0) {
                    ok = sv_wait(&bar_yf[par], ph_yf[par], fail);
                    ph_yf[par] ^= 1u;
                } else {
                    ok = sv_wait(&bar_x[2 * h + second - 1], ph_x, fail);
                    y = Yp;
                }
                if (!ok) break;
                sv_out32(v, w0, w4, y);
                Yp = y;
                __syncwarp();
                if (lane == 0) sv_arrive(h == 1 && second == 1 ? &bar_y[par] : &bar_x[2 * h + second]);
            }
            ph_x ^= 1u;
            if (!ok) s_fail = 1;
        }
    } else {
        // ---------------- row warps: two rows per thread ----------------
        // features of the next tile as soon as the input layer of the current
        // one has read its operand, then the spectra of the current one; the
        // tile's case sits in one of two shared slots, so that a new case can
        // be loaded while the previous one is still read
        const int rt = tid - 32 * (SV_WARPS + 1);
        uint32_t ph_a = 0u, ph_y[2] = {0u, 0u};
        int slot = 0, par = 0;
        bool ok = true;
        // the case of `tile` into slot `to` unless slot `from` already holds it
        auto locate = [&](int64_t tile, int from, int to) -> int {
            if (from >= 0 && tile >= sc[from].tile0 && tile < s_case_t1[from]) return from;
            sv_row_sync(true);  // every row warp is done with the case that `to` held
            if (rt < 32) {
                int lo = 0, hi = ncases - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (cases[mid].tile0 <= tile) lo = mid;
                    else hi = mid - 1;
                }
                const uint32_t *src = (const uint32_t *)(cases + lo);
                uint32_t *dst = (uint32_t *)&sc[to];
                for (int i = lane; i < (int)(sizeof(SurCase) / 4); i += 32) dst[i] = src[i];
                if (lane == 0) s_case_t1[to] = lo + 1 < ncases ? cases[lo + 1].tile0 : ntiles;
            }
            sv_row_sync(true);
            return to;
        };
        uint32_t mw[2] = {0u, 0u};  // mode words of this thread's rows (rt, rt + SV_ROWS) of the current tile
        if ((int64_t)blockIdx.x < ntiles) {
            slot = locate(blockIdx.x, -1, 0);
#pragma unroll
            for (int u = 0; u < 2; ++u) mw[u] = sv_mode_word(sc[slot], blockIdx.x, rt + u * SV_ROWS);
#pragma unroll 1
            for (int u = 0; u < 2; ++u)
                sv_features(sc[slot], blockIdx.x, rt + u * SV_ROWS, u == 0 ? mw[0] : mw[1], S.A0);
            tc_fence_proxy_async();
            sv_arrive(&bar_f);
        }
        for (int64_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, par ^= 1) {
            int next_slot = slot;
            uint32_t mw_next[2] = {0u, 0u};
            if (tile + gridDim.x < ntiles) {
                next_slot = locate(tile + gridDim.x, slot, slot ^ 1);
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    mw_next[u] = sv_mode_word(sc[next_slot], tile + gridDim.x, rt + u * SV_ROWS);
                ok = sv_wait(&bar_a, ph_a, fail);
                ph_a ^= 1u;
                if (ok) {
#pragma unroll 1
                    for (int u = 0; u < 2; ++u)
                        sv_features(sc[next_slot], tile + gridDim.x, rt + u * SV_ROWS,
                                    u == 0 ? mw_next[0] : mw_next[1], S.A0);
                    tc_fence_proxy_async();
                    sv_arrive(&bar_f);
                }
            }
            if (ok) ok = sv_wait(&bar_y[par], ph_y[par], fail);
            ok = sv_row_sync(ok);  // all or none go on: locate has the row warps meet
            if (!ok) break;
            ph_y[par] ^= 1u;
            const SurCase &c = sc[slot];
#pragma unroll 1
            for (int u = 0; u < 2; ++u) {
                const int rr = rt + u * SV_ROWS;
                const int64_t m = (tile - c.tile0) * 128 + rr;
                const float4 a = S.Yp[par][0][rr], b = S.Yp[par][1][rr];
                if (m < c.g.nsolved && !sv_in_band(c, u == 0 ? mw[0] : mw[1])) {
                    const float y[4] = {(a.x + b.x) + S.b4[0], (a.y + b.y) + S.b4[1], (a.z + b.z) + S.b4[2],
                                        (a.w + b.w) + S.b4[3]};
                    emit_spectrum(c.g, u == 0 ? mw[0] : mw[1], y, c.ax, c.ay, c.zm, c.inv_wind, c.ktop, c.utop, c.Xp,
                                  c.Xq);
                }
            }
            sv_arrive(&bar_yf[par]);
            slot = next_slot;
            mw[0] = mw_next[0];
            mw[1] = mw_next[1];
        }
        if (!ok) s_fail = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tc_tmem_free(tmem, 512);
}

inline unsigned blocks_for(int64_t n) { return (unsigned)((n + 255) / 256); }

}  // namespace

cudaError_t launch_sur_features(const SolveGeom &g, const uint32_t *modes, float ax, float ay, float zm, float s1,
                                float s2, float s3, float *X, int64_t npad, cudaStream_t st)
{
    if (npad <= 0) return cudaSuccess;
    sur_features_kernel<<<blocks_for(npad), 256, 0, st>>>(g, modes, ax, ay, zm, s1, s2, s3, X, npad);
    return cudaGetLastError();
}

cudaError_t launch_sur_exact(const SolveGeom &g, const uint32_t *modes, float ax, float ay, float zm,
                             const TransferCase *tc, const float4 *steps, float *Y, cudaStream_t st)
{
    if (g.nsolved <= 0) return cudaSuccess;
    sur_exact_kernel<<<blocks_for(g.nsolved), 256, 0, st>>>(g, modes, ax, ay, zm, tc, steps, Y);
    return cudaGetLastError();
}

cudaError_t launch_sur_serve(const SurCase *cases, int ncases, int64_t ntiles, const MlpServing &net, int *err,
                             int nsm, cudaStream_t st)
{
    if (ntiles <= 0 || ncases <= 0) return cudaSuccess;
    static uint64_t attr = 0;
    if (first_on_device(attr)) {
        cudaError_t e = cudaFuncSetAttribute(sur_serve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(SvSmem));
        if (e != cudaSuccess) {
            attr = 0;
            return e;
        }
    }
    const int grid = (int)std::min<int64_t>(ntiles, std::max(nsm, 1));
    sur_serve_kernel<<<grid, SV_THREADS, sizeof(SvSmem), st>>>(cases, ncases, ntiles, net, err);
    return cudaGetLastError();
}

cudaError_t launch_sur_spectra(const SolveGeom &g, const uint32_t *modes, const float *Y, float ax, float ay,
                               float zm, float inv_wind, float ktop, float utop, float2 *Xp, float2 *Xq,
                               cudaStream_t st)
{
    if (g.nsolved <= 0) return cudaSuccess;
    sur_spectra_kernel<<<blocks_for(g.nsolved), 256, 0, st>>>(g, modes, Y, ax, ay, zm, inv_wind, ktop, utop, Xp,
                                                              Xq);
    return cudaGetLastError();
}
