// Device kernels of the steady-state transport solve.
//
//   sweep64_kernel     ivp_solver (src/bldfm/solver.py:307-374), both shooting IVPs
//   combine64_kernel   alpha + level combination + shift (solver.py:228-235, 253-262)
//   trapezoid_kernel   k = 0 mode (solver.py:237-251)
//   analytic64_kernel  constant-profile closed form (solver.py:193-202)
//   riccati32_kernel   FP32 invariant-imbedding sweep of the same discrete BVP
//   fwd_rows / fwd_cols   truncated forward FFT of the source (solver.py:136-145)
//   out_cols / out_rows   un-truncate + output FFT + crop (solver.py:264-290)
//
// FP64 kernels reproduce the reference's numpy rounding: every operation is an
// explicit round-to-nearest intrinsic (no contraction), and complex products use
// numpy's x86-64 pattern re = fma(ar, br, -(ai*bi)), im = fma(ar, bi, ai*br).
#include "devattr.h"
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "common.h"
#include "devmath.cuh"
#include "fft_core.cuh"
#include "kernels.h"
#include "sweep32.cuh"
#include "fft_passes.cuh"

#define LAUNCH_CHECK() (cudaGetLastError())

// ---------------------------------------------------------------------------
// FP64 shooting sweep
// ---------------------------------------------------------------------------
// FP64 instructions of this GPU take 16 clocks per warp and SM as an FMA of
// three registers and 19 as an addition or a multiplication (0.628 against
// 0.529 T lanes/s, measured with register operands; an FMA with a constant or
// uniform operand takes 19 too).  a + b = fma(a, 1, b) and a b = fma(a, b, -0)
// round, and sign their zeros, exactly as the addition and the product do, so
// the sweep issues nothing but FMAs, the 1 and the -0 in registers the
// compiler cannot see through (read from shared memory).
struct FmaArith {
    double one, mz, two9;
    __device__ __forceinline__ double add(double a, double b) const { return __fma_rn(a, one, b); }
    __device__ __forceinline__ double sub(double a, double b) const { return __fma_rn(b, -one, a); }
    __device__ __forceinline__ double mul(double a, double b) const { return __fma_rn(a, b, mz); }
    __device__ __forceinline__ double2 cmul(double2 a, double2 b) const
    {
        return make_double2(__fma_rn(a.x, b.x, -mul(a.y, b.y)), __fma_rn(a.x, b.y, mul(a.y, b.x)));
    }
    // a b for a = -n
    __device__ __forceinline__ double2 cmul_neg(double2 n, double2 b) const
    {
        return make_double2(__fma_rn(-n.x, b.x, mul(n.y, b.y)), __fma_rn(-n.x, b.y, -mul(n.y, b.x)));
    }
    __device__ __forceinline__ double2 cadd(double2 a, double2 b) const
    {
        return make_double2(add(a.x, b.x), add(a.y, b.y));
    }
};

// both shooting states of one mode
struct Shoot {
    double2 p1, q1, p2, q2;
};

// Items of the paired sweep (NM = 2): the modes (kx, ky) and (kx, -ky) of a
// column share T's real part and what follows from it (Re a, Re b, Re T dz and
// the four products inside T): 62 FP64 instructions a mode and step instead of
// 68.  In the mode list's order, column 0 holds its C0 rows from row 1 on,
// columns 1 .. F every row, the columns after them one row each (even nly).
struct SweepItems {
    int C0, F, I, n;  // I items per full column: rows 0 .. nly / 2; n items in all
};

__host__ __device__ inline SweepItems sweep_items(int nlx, int nly)
{
    SweepItems s;
    s.C0 = freq_max(nly) + (nly % 2 == 0 ? 1 : 0);
    s.F = nlx / 2;
    s.I = nly / 2 + 1;
    s.n = s.C0 + s.F * s.I + (nly % 2 == 0 ? nlx - 1 - s.F : 0);
    return s;
}

// column, row and list index of item i; its partner's list index or -1
__device__ __forceinline__ void sweep_item(const SweepItems &s, int nly, int i, int &c, int &r, int64_t &m0,
                                           int64_t &m1)
{
    m1 = -1;
    if (i < s.C0) {
        c = 0;
        r = i + 1;
        m0 = i;
        return;
    }
    const int j = i - s.C0;
    if (j < s.F * s.I) {
        c = 1 + j / s.I;
        r = j - (c - 1) * s.I;
        const int64_t base = s.C0 + (int64_t)(c - 1) * nly;
        m0 = base + r;
        if (r > 0 && 2 * r != nly) m1 = base + nly - r;
        return;
    }
    c = s.F + 1 + (j - s.F * s.I);
    r = nly / 2;
    m0 = s.C0 + (int64_t)s.F * nly + (j - s.F * s.I);
}

#define SWEEP64_THREADS 512

// Items of a thread of the FP64 sweeps: warps of 32 items, dealt to the blocks
// (one per SM) in turn, so that every SM holds the same number to within one.
struct SweepWarp {
    int64_t first, step;
    __device__ __forceinline__ SweepWarp()
    {
        first = 32 * ((int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) + (threadIdx.x & 31);
        step = (int64_t)blockDim.x * gridDim.x;
    }
};

// NM modes per thread (2: the items above).  Writes per mode: top states
// (p1,q1,p2,q2) and the same four states at every snapshot slot.
//   snap layout: [(slot * 4 + j) * nsolved + m],  top layout: [j * nsolved + m]
template <int NM>
__global__ void __launch_bounds__(SWEEP64_THREADS) sweep64_kernel(SolveGeom g, const double *__restrict__ lvtab,
                                                      const int *__restrict__ slot_of_step,
                                                      const uint32_t *__restrict__ modes,
                                                      const double2 *__restrict__ q0spec,
                                                      double2 *__restrict__ snap, double2 *__restrict__ top,
                                                      int *err)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t bar;
    __shared__ double s_one[4];
    double *s_lv = (double *)smem_raw;
    const int L = g.nz - 1;
    int *s_slot = (int *)(s_lv + (size_t)L * BLDFM_LV64);
    if (threadIdx.x < 4) s_one[threadIdx.x] = threadIdx.x < 2 ? 1.0 : -0.0;
    if (L > 0) {
        if (!bulk_load_to_smem(s_lv, lvtab, (uint32_t)((size_t)L * BLDFM_LV64 * sizeof(double)), &bar, err))
            return;
    }
    for (int i = threadIdx.x; i < g.nz; i += blockDim.x) s_slot[i] = slot_of_step[i];
    __syncthreads();
    const FmaArith F = {s_one[threadIdx.x & 1], s_one[2 + (threadIdx.x & 1)], 0.0};

    const int64_t ns = g.nsolved;
    const SweepItems si = sweep_items(g.nlx, g.nly);
    const int64_t n = NM == 2 ? si.n : ns;
    const SweepWarp sw;
    for (int64_t it = sw.first; it < n; it += sw.step) {
        int r, c;
        int64_t m[2] = {it, -1};
        if (NM == 2) {
            sweep_item(si, g.nly, (int)it, c, r, m[0], m[1]);
        } else {
            bool paired;
            unpack_mode(modes[it], r, c, paired);
        }
        const double lx = wavenumber(freq_of_index(c, g.nlx), g.valx, g.lx_scale);
        const double ly = wavenumber(freq_of_index(r, g.nly), g.valy, g.ly_scale);
        const double lx2 = __dmul_rn(lx, lx), ly2 = __dmul_rn(ly, ly);
        Shoot S[NM];
#pragma unroll
        for (int u = 0; u < NM; ++u) {
            S[u].p1 = make_double2(1.0, 0.0);
            S[u].q1 = S[u].p2 = make_double2(0.0, 0.0);
            S[u].q2 = q0spec ? q0spec[(size_t)c * g.nly + (u == 0 || r == 0 ? r : g.nly - r)]
                             : make_double2(g.q0dc_fp, 0.0);
        }
        auto store = [&](double2 *o, int u) {
            o += m[u];
            o[0] = S[u].p1;
            o[ns] = S[u].q1;
            o[2 * ns] = S[u].p2;
            o[3 * ns] = S[u].q2;
        };
        for (int i = 0; i < L; ++i) {
            const int s = s_slot[i];
            if (s >= 0) {
                store(snap + (size_t)s * 4 * ns, 0);
                if (NM == 2 && m[NM - 1] >= 0) store(snap + (size_t)s * 4 * ns, NM - 1);
            }
            const double *lv = s_lv + (size_t)i * BLDFM_LV64;
            // T = -(Kx Lx^2 + Ky Ly^2) - 1j u Lx - 1j v Ly = -(tx + 1j ty)
            const double tx = F.add(F.mul(lv[LV_KX], lx2), F.mul(lv[LV_KY], ly2));
            const double ul = F.mul(lv[LV_U], lx), vl = F.mul(lv[LV_V], ly);
            // real parts of a = d = 1 - 0.5 Kzinv T dz^2 and
            // b = -Kzinv dz - 1/6 Kzinv^2 T dz^3; T dz
            const double ax = F.add(F.mul(F.mul(lv[LV_S1], tx), lv[LV_H2]), F.one);
            const double bx = F.add(F.mul(F.mul(lv[LV_S2], tx), lv[LV_H3]), lv[LV_S3]);
            const double txh = F.mul(tx, lv[LV_H]);
#pragma unroll
            for (int u = 0; u < NM; ++u) {
                const double ty = u == 0 ? F.add(ul, vl) : F.sub(ul, vl);
                const double2 a = make_double2(ax, F.mul(F.mul(lv[LV_S1], ty), lv[LV_H2]));
                const double2 b = make_double2(bx, F.mul(F.mul(lv[LV_S2], ty), lv[LV_H3]));
                // c = T dz - 1/6 Kzinv T^2 dz^3, negated
                const double2 T2 = F.cmul(make_double2(tx, ty), make_double2(tx, ty));
                const double2 cn =
                    make_double2(F.add(F.mul(F.mul(lv[LV_S4], T2.x), lv[LV_H3]), txh),
                                 F.add(F.mul(F.mul(lv[LV_S4], T2.y), lv[LV_H3]), F.mul(ty, lv[LV_H])));
                Shoot &x = S[u];
                const double2 np1 = F.cadd(F.cmul(a, x.p1), F.cmul(b, x.q1));
                const double2 nq1 = F.cadd(F.cmul_neg(cn, x.p1), F.cmul(a, x.q1));
                const double2 np2 = F.cadd(F.cmul(a, x.p2), F.cmul(b, x.q2));
                const double2 nq2 = F.cadd(F.cmul_neg(cn, x.p2), F.cmul(a, x.q2));
                x.p1 = np1;
                x.q1 = nq1;
                x.p2 = np2;
                x.q2 = nq2;
            }
        }
        const int s = s_slot[g.nz - 1];
#pragma unroll
        for (int u = 0; u < NM; ++u) {
            if (u > 0 && m[u] < 0) break;
            if (s >= 0) store(snap + (size_t)s * 4 * ns, u);
            store(top, u);
        }
    }
}

// The sweep of a small solve, which leaves the SMs with fewer than four warps:
// four lanes per mode, lane 2 k + 0 / 1 for the p / q of shooting state k, so
// that a lane's chain is 33 instructions a step instead of 68 (every operation
// and rounding of sweep64_kernel's, B = b or -c).  96^2 modes over 104 levels:
// 230 us with a mode per thread, 138 so.
__global__ void __launch_bounds__(SWEEP64_THREADS) sweep64_lanes_kernel(SolveGeom g, const double *__restrict__ lvtab,
                                                                        const int *__restrict__ slot_of_step,
                                                                        const uint32_t *__restrict__ modes,
                                                                        const double2 *__restrict__ q0spec,
                                                                        double2 *__restrict__ snap,
                                                                        double2 *__restrict__ top, int *err)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t bar;
    __shared__ double s_one[4];
    double *s_lv = (double *)smem_raw;
    const int L = g.nz - 1;
    int *s_slot = (int *)(s_lv + (size_t)L * BLDFM_LV64);
    if (threadIdx.x < 4) s_one[threadIdx.x] = threadIdx.x < 2 ? 1.0 : -0.0;
    if (L > 0) {
        if (!bulk_load_to_smem(s_lv, lvtab, (uint32_t)((size_t)L * BLDFM_LV64 * sizeof(double)), &bar, err))
            return;
    }
    for (int i = threadIdx.x; i < g.nz; i += blockDim.x) s_slot[i] = slot_of_step[i];
    __syncthreads();
    const FmaArith F = {s_one[threadIdx.x & 1], s_one[2 + (threadIdx.x & 1)], 0.0};

    const int64_t ns = g.nsolved;
    const SweepWarp sw;
    const int lane = threadIdx.x & 31, part = lane & 3;  // p1, q1, p2, q2
    const bool isq = part & 1;
    for (int64_t it = sw.first; it - lane < 4 * ns; it += sw.step) {  // whole warps: the lanes exchange p and q
        const bool on = it < 4 * ns;
        const int64_t m = on ? it >> 2 : ns - 1;
        int r, c;
        bool paired;
        unpack_mode(modes[m], r, c, paired);
        const double lx = wavenumber(freq_of_index(c, g.nlx), g.valx, g.lx_scale);
        const double ly = wavenumber(freq_of_index(r, g.nly), g.valy, g.ly_scale);
        const double lx2 = __dmul_rn(lx, lx), ly2 = __dmul_rn(ly, ly);
        double2 x = make_double2(part == 0 ? 1.0 : 0.0, 0.0);
        if (part == 3) x = q0spec ? q0spec[(size_t)c * g.nly + r] : make_double2(g.q0dc_fp, 0.0);
        for (int i = 0; i < L; ++i) {
            const int s = s_slot[i];
            if (s >= 0 && on) snap[((size_t)s * 4 + part) * ns + m] = x;
            const double *lv = s_lv + (size_t)i * BLDFM_LV64;
            const double tx = F.add(F.mul(lv[LV_KX], lx2), F.mul(lv[LV_KY], ly2));
            const double ty = F.add(F.mul(lv[LV_U], lx), F.mul(lv[LV_V], ly));
            const double2 a = make_double2(F.add(F.mul(F.mul(lv[LV_S1], tx), lv[LV_H2]), F.one),
                                           F.mul(F.mul(lv[LV_S1], ty), lv[LV_H2]));
            const double2 T2 = F.cmul(make_double2(tx, ty), make_double2(tx, ty));
            const double k = isq ? lv[LV_S4] : lv[LV_S2];
            const double vx = F.mul(tx, lv[LV_H]), vy = F.mul(ty, lv[LV_H]);
            double2 b = make_double2(
                F.add(F.mul(F.mul(k, isq ? T2.x : tx), lv[LV_H3]), isq ? vx : lv[LV_S3]),
                F.add(F.mul(F.mul(k, isq ? T2.y : ty), lv[LV_H3]), isq ? vy : F.mz));
            if (isq) b = make_double2(-b.x, -b.y);
            double2 o;
            o.x = __shfl_xor_sync(0xffffffffu, x.x, 1);
            o.y = __shfl_xor_sync(0xffffffffu, x.y, 1);
            x = F.cadd(F.cmul(a, x), F.cmul(b, o));
        }
        if (!on) continue;
        const int s = s_slot[g.nz - 1];
        if (s >= 0) snap[((size_t)s * 4 + part) * ns + m] = x;
        top[part * ns + m] = x;
    }
}

// ---------------------------------------------------------------------------
// FP64 combination: alpha, levels, complex64 rounding, phase shift, mirror
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) combine64_kernel(SolveGeom g, const uint32_t *__restrict__ modes,
                                                        const double2 *__restrict__ eig,
                                                        const double2 *__restrict__ snap,
                                                        const double2 *__restrict__ top, double2 *__restrict__ Xp,
                                                        double2 *__restrict__ Xq)
{
    const int64_t ns = g.nsolved;
    const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= ns) return;
    int r, c;
    bool paired;
    unpack_mode(modes[m], r, c, paired);
    const int kx = freq_of_index(c, g.nlx), ky = freq_of_index(r, g.nly);
    // alpha = -(q2 - Kz eig p2) / (q1 - Kz eig p1)
    const double2 e = eig[m];
    const double2 keig = make_double2(__dmul_rn(g.kz_top, e.x), __dmul_rn(g.kz_top, e.y));
    double2 num = np_csub(top[3 * ns + m], np_cmul(keig, top[2 * ns + m]));
    const double2 den = np_csub(top[ns + m], np_cmul(keig, top[m]));
    num.x = -num.x;
    num.y = -num.y;
    const double2 alpha = np_cdiv(num, den);

    double2 shift = make_double2(1.0, 0.0);
    if (g.do_shift) {
        const double lx = wavenumber(kx, g.valx, g.lx_scale);
        const double ly = wavenumber(ky, g.valy, g.ly_scale);
        const double th = __dadd_rn(__dmul_rn(lx, g.sx), __dmul_rn(ly, g.sy));
        double sn, cs;
        sincos(th, &sn, &cs);
        shift = make_double2(cs, sn);
    }
    const int rm = paired ? index_of_freq(-ky, g.nly) : 0;
    const int cm = paired ? index_of_freq(-kx, g.nlx) : 0;
    for (int s = 0; s < g.nsnap; ++s) {
        const double2 *sp = snap + (size_t)s * 4 * ns + m;
        double2 p = np_cadd(np_cmul(alpha, sp[0]), sp[2 * ns]);
        double2 q = np_cadd(np_cmul(alpha, sp[ns]), sp[3 * ns]);
        if (g.precision == 0) {
            p = round_c64(p);
            q = round_c64(q);
        }
        if (g.do_shift) {
            p = np_cmul(p, shift);
            q = np_cmul(q, shift);
        }
        Xp[spec_idx(g, s, r, c)] = p;
        Xq[spec_idx(g, s, r, c)] = q;
        if (paired) {
            Xp[spec_idx(g, s, rm, cm)] = make_double2(p.x, -p.y);
            Xq[spec_idx(g, s, rm, cm)] = make_double2(q.x, -q.y);
        }
    }
}

// ---------------------------------------------------------------------------
// k = 0 mode: trapezoid rule, one thread.  lvtab column LV_PAD holds
// w_i = 0.5/Kz[i] + 0.5/Kz[i+1], column LV_H holds dz[i].
// ---------------------------------------------------------------------------
// k = 0 mode when q0 lives on the device (dispersion mode): writes the
// reference's trapezoid values (solver.py:237-251) into dc[2 s] (p), dc[2 s + 1]
// (q).  The terms (q0 dz_i) w_i are independent and computed in parallel; the
// running difference keeps the reference's order on one thread.
// dcp (may be NULL): DC_PARTS partial FP64 sums of the source field
// (dc_partial_kernel); the k = 0 source value is then their sum / (nxe nye)
// in FP64 instead of the transform's k = 0 output.
__device__ __forceinline__ void trapezoid_values(const SolveGeom &g, const double *__restrict__ lvtab,
                                                 const int *__restrict__ slot_of_step, double2 q0, double p000,
                                                 double2 *__restrict__ dc, unsigned char *smem_raw)
{
    double2 *term = (double2 *)smem_raw;
    int *sl = (int *)(term + (g.nz > 1 ? g.nz - 1 : 1));
    const bool single = g.precision == 0;
    const double2 qs = single ? round_c64(q0) : q0;
    for (int s = threadIdx.x; s < g.nlvls; s += blockDim.x) {
        dc[2 * s + 1] = qs;
        if (s > 0) dc[2 * s] = make_double2(0.0, 0.0);
    }
    for (int i = threadIdx.x; i < g.nz - 1; i += blockDim.x) {
        const double dz = lvtab[(size_t)i * BLDFM_LV64 + LV_H];
        const double w = lvtab[(size_t)i * BLDFM_LV64 + LV_PAD];
        term[i] = make_double2(__dmul_rn(__dmul_rn(q0.x, dz), w), __dmul_rn(__dmul_rn(q0.y, dz), w));
    }
    for (int i = threadIdx.x; i < g.nz; i += blockDim.x) sl[i] = slot_of_step[i];
    __syncthreads();
    if (threadIdx.x != 0) return;
    dc[0] = make_double2(single ? (double)__double2float_rn(p000) : p000, 0.0);
    if (g.analytic) return;
    double2 p00 = make_double2(p000, 0.0);
    for (int i = 0; i < g.nz - 1; ++i) {
        const int s = sl[i];
        if (s >= 0) dc[2 * s] = single ? round_c64(p00) : p00;
        p00.x = __dsub_rn(p00.x, term[i].x);
        p00.y = __dsub_rn(p00.y, term[i].y);
    }
    const int s = sl[g.nz - 1];
    if (s >= 0) dc[2 * s] = single ? round_c64(p00) : p00;
}

template <typename C>
__global__ void __launch_bounds__(256) trapezoid_kernel(SolveGeom g, const double *__restrict__ lvtab,
                                                        const int *__restrict__ slot_of_step,
                                                        const C *__restrict__ q0spec, double p000,
                                                        double2 *__restrict__ dc, const double *__restrict__ dcp)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 q0 = make_double2((double)q0spec[0].x, (double)q0spec[0].y);
    if (dcp) {
        double sum = 0.0;
        for (int b = 0; b < DC_PARTS; ++b) sum += dcp[b];
        q0 = make_double2(sum * g.inv_nxe * g.inv_nye, 0.0);
    }
    trapezoid_values(g, lvtab, slot_of_step, q0, p000, dc, smem_raw);
}

// the k = 0 values of a batch's dispersion cases, one block per case
__global__ void __launch_bounds__(256) trapezoid_batch_kernel(const FwdCase *__restrict__ cases)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const FwdCase &c = cases[blockIdx.x];
    double sum = 0.0;
    for (int b = 0; b < DC_PARTS; ++b) sum += c.dcp[b];
    trapezoid_values(c.g, c.lv64, c.slot, make_double2(sum * c.g.inv_nxe * c.g.inv_nye, 0.0), c.p000, c.dc, smem_raw);
}

// ---------------------------------------------------------------------------
// analytic branch (constant profiles, one output level)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) analytic64_kernel(SolveGeom g, const uint32_t *__restrict__ modes,
                                                         const double2 *__restrict__ eig,
                                                         const double2 *__restrict__ q0spec, double kzinv,
                                                         double hlev, double2 *__restrict__ Xp,
                                                         double2 *__restrict__ Xq)
{
    const int64_t ns = g.nsolved;
    const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= ns) return;
    int r, c;
    bool paired;
    unpack_mode(modes[m], r, c, paired);
    const int kx = freq_of_index(c, g.nlx), ky = freq_of_index(r, g.nly);
    const double2 e = eig[m];
    const double2 q0 = q0spec ? q0spec[(size_t)c * g.nly + r] : make_double2(g.q0dc_fp, 0.0);
    // tfftq = q0 * exp(-eig * h)
    const double er = __dmul_rn(-e.x, hlev), ei = __dmul_rn(-e.y, hlev);
    double sn, cs;
    sincos(ei, &sn, &cs);
    const double ex = exp(er);
    double2 q = np_cmul(q0, make_double2(ex * cs, ex * sn));
    if (g.precision == 0) q = round_c64(q);
    // tfftp = tfftq * Kzinv / eig
    double2 p = np_cdiv(make_double2(__dmul_rn(q.x, kzinv), __dmul_rn(q.y, kzinv)), e);
    if (g.precision == 0) p = round_c64(p);
    if (g.do_shift) {
        const double lx = wavenumber(kx, g.valx, g.lx_scale);
        const double ly = wavenumber(ky, g.valy, g.ly_scale);
        const double th = __dadd_rn(__dmul_rn(lx, g.sx), __dmul_rn(ly, g.sy));
        double s2, c2;
        sincos(th, &s2, &c2);
        const double2 sh = make_double2(c2, s2);
        p = np_cmul(p, sh);
        q = np_cmul(q, sh);
    }
    Xp[spec_idx(g, 0, r, c)] = p;
    Xq[spec_idx(g, 0, r, c)] = q;
    if (paired) {
        const int rm = index_of_freq(-ky, g.nly), cm = index_of_freq(-kx, g.nlx);
        Xp[spec_idx(g, 0, rm, cm)] = make_double2(p.x, -p.y);
        Xq[spec_idx(g, 0, rm, cm)] = make_double2(q.x, -q.y);
    }
}

// analytic k = 0 (dispersion mode, q0 on the device): p = p000 - q0 Kzinv h, q = q0
__global__ void analytic_dc_kernel(SolveGeom g, const double2 *__restrict__ q0spec, double p000, double kzinv,
                                   double hlev, double2 *__restrict__ dc)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double2 q0 = q0spec[0];
    double2 p = make_double2(__dsub_rn(p000, __dmul_rn(__dmul_rn(q0.x, kzinv), hlev)),
                             __dsub_rn(0.0, __dmul_rn(__dmul_rn(q0.y, kzinv), hlev)));
    double2 q = q0;
    if (g.precision == 0) {
        p = round_c64(p);
        q = round_c64(q);
    }
    dc[0] = p;
    dc[1] = q;
}

// One thread per solved mode, grid-stride.
template <bool ISO, bool SINGLE>
__global__ void __launch_bounds__(256) riccati32_kernel(SolveGeom g, const float *__restrict__ lv32,
                                                        const int *__restrict__ slot_of_step,
                                                        const uint32_t *__restrict__ modes,
                                                        const float2 *__restrict__ q0spec,
                                                        float *__restrict__ scratch, float2 *__restrict__ Xp,
                                                        float2 *__restrict__ Xq, float ax, float ay, int *err)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t bar;
    float *s_lv = (float *)smem_raw;
    const int L = g.nz - 1;
    int *s_slot = (int *)(s_lv + (size_t)L * BLDFM_LV32);
    if (L > 0) {
        if (!bulk_load_to_smem(s_lv, lv32, (uint32_t)((size_t)L * BLDFM_LV32 * sizeof(float)), &bar, err)) return;
    }
    for (int i = threadIdx.x; i < g.nz; i += blockDim.x) s_slot[i] = slot_of_step[i];
    __syncthreads();
    const int64_t ns = g.nsolved;
    if (SINGLE) {
        // two modes per thread (m and m + blockDim.x) in the lanes of packed f32x2 operations
        const int64_t step = 2 * (int64_t)gridDim.x * blockDim.x;
        for (int64_t m = 2 * (int64_t)blockIdx.x * blockDim.x + threadIdx.x; m < ns; m += step) {
            const int64_t mb = m + blockDim.x < ns ? m + blockDim.x : -1;
            ricc_mode_pair<ISO>(g, s_lv, modes, q0spec, Xp, Xq, ax, ay, m, mb);
        }
    } else {
        for (int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; m < ns; m += (int64_t)gridDim.x * blockDim.x)
            ricc_mode<ISO, SINGLE>(g, s_lv, s_slot, modes, q0spec, scratch, Xp, Xq, ax, ay, m);
    }
}

// ---------------------------------------------------------------------------
// FP64 invariant-imbedding sweep (accurate mode)
// ---------------------------------------------------------------------------
// The FP32 kernel's recursion in FP64 with exact division: the solution of the
// reference's discrete problem without the shooting method's cancellation.
__device__ __forceinline__ double2 csqrt_d(double2 w)
{
    const double x = w.x, y = w.y;
    const double t = sqrt(0.5 * (fabs(x) + hypot(x, y)));
    if (t == 0.0) return make_double2(0.0, 0.0);
    if (x >= 0.0) return make_double2(t, y / (2.0 * t));
    return make_double2(fabs(y) / (2.0 * t), copysign(t, y));
}

__device__ __forceinline__ double2 dc_mul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}

// Accurate FP64 sweep: invariant imbedding in its homogeneous form.  The ratio
// R_i = p_i / q_i of the decaying solution is N_i / D_i with
//   N <- a N - b D,   D <- a D - c N
// (16 FMAs a step where the update of R with its reciprocal takes 22), and the
// flux factors telescope: q_j / q_0 = (D_j / D_0) prod_{i<j} det_i with
// det_i = a^2 - b c.  With w = a - 1 the step's coefficients are
//   a = 1 + w,  b = B0 - (B0 / 3) w,  c = g (w + w^2 / 3),  g = 2 / B0,
//   det = 1 + w^2 + (2/9) w^3,
// w = (A Kx lx^2 + A Ky ly^2) + i (A u lx + A v ly), A = dz^2 / (2 Kz),
// B0 = -dz / Kz.  The FP64 pipe bounds it (FmaArith above): 27 instructions a
// mode and step above the highest output level and 36.5 below it for a pair of
// modes (kx, +-ky) per thread, 30 and 40 alone; the ratio form took 38 and 46,
// a third of them additions and multiplications.  States and determinant are
// rescaled by powers of two every 4 steps (integer arithmetic on the exponent).
enum { RT_AKX, RT_AKY, RT_AU, RT_AV, RT_B0, RT_B1, RT_G, RT_G3, RT_N };
#define RICC64_SMEM (200 * 1024)  // dynamic shared memory the kernel is set up for

// exponent of the largest of n values (0 for zeros and non-finite values)
__device__ __forceinline__ int top_exponent(const double *v, int n)
{
    int e = 0;
#pragma unroll
    for (int k = 0; k < n; ++k) e = max(e, (__double2hiint(v[k]) >> 20) & 0x7ff);
    return e == 0 || e == 0x7ff ? 0 : e - 1023;
}
// v 2^-e (values outside the normal range, before or after, become zero)
__device__ __forceinline__ double scale_down(double v, int e)
{
    const int hi = __double2hiint(v), x = (hi >> 20) & 0x7ff;
    if (x == 0x7ff) return v;
    return x == 0 || x - e <= 0 ? 0.0 : __hiloint2double(hi - e * (1 << 20), __double2loint(v));
}

struct RiccState {
    double n[4];  // N, D (re, im)
    double2 P;    // product of det_i below the highest output level
    int E, EP;    // their powers of two
};

template <bool SINGLE, int NM>
__global__ void __launch_bounds__(SWEEP64_THREADS) riccati64_kernel(SolveGeom g, const double *__restrict__ lvtab,
                                                        const int *__restrict__ slot_of_step,
                                                        const uint32_t *__restrict__ modes,
                                                        const double2 *__restrict__ q0spec,
                                                        double *__restrict__ scratch, double2 *__restrict__ Xp,
                                                        double2 *__restrict__ Xq)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double s_one[6];
    double *s_rt = (double *)smem_raw;
    const int L = g.nz - 1;
    int *s_slot = (int *)(s_rt + (size_t)L * RT_N);
    if (threadIdx.x < 6) s_one[threadIdx.x] = threadIdx.x < 2 ? 1.0 : threadIdx.x < 4 ? -0.0 : 2.0 / 9.0;
    for (int i = threadIdx.x; i < L; i += blockDim.x) {
        const double *lv = lvtab + (size_t)i * BLDFM_LV64;
        double *o = s_rt + (size_t)i * RT_N;
        const double A = lv[LV_S1] * lv[LV_H2], B0 = lv[LV_S3], G = 2.0 / B0;
        o[RT_AKX] = A * lv[LV_KX];
        o[RT_AKY] = A * lv[LV_KY];
        o[RT_AU] = A * lv[LV_U];
        o[RT_AV] = A * lv[LV_V];
        o[RT_B0] = B0;
        o[RT_B1] = -B0 / 3.0;
        o[RT_G] = G;
        o[RT_G3] = G / 3.0;
    }
    for (int i = threadIdx.x; i < g.nz; i += blockDim.x) s_slot[i] = slot_of_step[i];
    __syncthreads();
    const FmaArith F = {s_one[threadIdx.x & 1], s_one[2 + (threadIdx.x & 1)], s_one[4 + (threadIdx.x & 1)]};
    const int jmax = g.jmax;
    const int64_t ns = g.nsolved;
    const SweepItems si = sweep_items(g.nlx, g.nly);
    const int64_t n = NM == 2 ? si.n : ns;
    const SweepWarp sw;
    for (int64_t it = sw.first; it < n; it += sw.step) {
        int r, c;
        int64_t m[2] = {it, -1};
        if (NM == 2) {
            sweep_item(si, g.nly, (int)it, c, r, m[0], m[1]);
        } else {
            bool paired;
            unpack_mode(modes[it], r, c, paired);
        }
        const int kx = freq_of_index(c, g.nlx), ky = freq_of_index(r, g.nly);
        const double lx = wavenumber(kx, g.valx, g.lx_scale), ly = wavenumber(ky, g.valy, g.ly_scale);
        const double lx2 = lx * lx, ly2 = ly * ly;
        RiccState S[NM];
#pragma unroll
        for (int u = 0; u < NM; ++u) {
            const double l = u == 0 ? ly : -ly;
            const double2 eg =
                csqrt_d(make_double2(fma(g.kxk_top, lx2, g.kyk_top * ly2), fma(g.uk_top, lx, g.vk_top * l)));
            const double2 ke = make_double2(g.kz_top * eg.x, g.kz_top * eg.y);
            const double kn = 1.0 / fma(ke.x, ke.x, ke.y * ke.y);
            S[u].n[0] = ke.x * kn;
            S[u].n[1] = -ke.y * kn;
            S[u].n[2] = 1.0;
            S[u].n[3] = 0.0;
            S[u].P = make_double2(1.0, 0.0);
            S[u].E = S[u].EP = 0;
        }
        // one step down; DET: with the determinant
        auto step = [&](int i, auto det) {
            constexpr bool DET = decltype(det)::value;
            const double *t = s_rt + (size_t)i * RT_N;
            const double wr = __fma_rn(t[RT_AKX], lx2, F.mul(t[RT_AKY], ly2));
            const double ul = F.mul(t[RT_AU], lx), vl = F.mul(t[RT_AV], ly);
            const double ar = F.add(wr, F.one), br = __fma_rn(t[RT_B1], wr, t[RT_B0]), gr = F.mul(t[RT_G], wr),
                         w2 = F.mul(wr, wr), w9 = DET ? __fma_rn(F.two9, wr, F.one) : 0.0;
#pragma unroll
            for (int u = 0; u < NM; ++u) {
                const double wi = u == 0 ? F.add(ul, vl) : F.sub(ul, vl);
                const double bi = F.mul(t[RT_B1], wi);
                const double sr = __fma_rn(-wi, wi, w2), h = F.mul(wr, wi);  // w^2 = sr + 2 i h
                const double cr = __fma_rn(t[RT_G3], sr, gr);
                const double h2 = F.add(h, h);
                const double ci = __fma_rn(t[RT_G3], h2, F.mul(t[RT_G], wi));
                double *v = S[u].n;
                const double Nr = v[0], Ni = v[1], Dr = v[2], Di = v[3];
                v[0] = __fma_rn(ar, Nr, __fma_rn(-wi, Ni, __fma_rn(-br, Dr, F.mul(bi, Di))));
                v[1] = __fma_rn(ar, Ni, __fma_rn(wi, Nr, __fma_rn(-br, Di, -F.mul(bi, Dr))));
                v[2] = __fma_rn(ar, Dr, __fma_rn(-wi, Di, __fma_rn(-cr, Nr, F.mul(ci, Ni))));
                v[3] = __fma_rn(ar, Di, __fma_rn(wi, Dr, __fma_rn(-cr, Ni, -F.mul(ci, Nr))));
                if (DET) {
                    // det - 1 = w^2 (1 + (2/9) w)
                    const double wi9 = F.mul(F.two9, wi);
                    const double er = __fma_rn(sr, w9, -F.mul(h2, wi9)), ei = __fma_rn(sr, wi9, F.mul(h2, w9));
                    const double2 P = S[u].P;
                    S[u].P.x = __fma_rn(P.x, er, __fma_rn(-P.y, ei, P.x));
                    S[u].P.y = __fma_rn(P.x, ei, __fma_rn(P.y, er, P.y));
                }
            }
        };
        auto rescale = [&](bool det) {
#pragma unroll
            for (int u = 0; u < NM; ++u) {
                const int e = top_exponent(S[u].n, 4);
#pragma unroll
                for (int k = 0; k < 4; ++k) S[u].n[k] = scale_down(S[u].n[k], e);
                S[u].E += e;
                if (det) {
                    const double pv[2] = {S[u].P.x, S[u].P.y};
                    const int ep = top_exponent(pv, 2);
                    S[u].P = make_double2(scale_down(pv[0], ep), scale_down(pv[1], ep));
                    S[u].EP += ep;
                }
            }
        };
        int i = L - 1;
        for (; i >= jmax; --i) {
            step(i, std::false_type());
            if ((i & 3) == 0) rescale(false);
        }
        RiccState J[NM];  // the states at the highest output level
#pragma unroll
        for (int u = 0; u < NM; ++u) J[u] = S[u];
        // scratch of an output slot: (N, D) / P and its power of two
        auto keep = [&](int s) {
#pragma unroll
            for (int u = 0; u < NM; ++u) {
                if (m[u] < 0) continue;
                double *o = scratch + (size_t)s * 5 * ns + m[u];
                const double2 P = S[u].P;
                const double pn = 1.0 / fma(P.x, P.x, P.y * P.y);
                const double2 inv = make_double2(P.x * pn, -P.y * pn);
                const double2 N = dc_mul(make_double2(S[u].n[0], S[u].n[1]), inv),
                              D = dc_mul(make_double2(S[u].n[2], S[u].n[3]), inv);
                o[0] = N.x;
                o[ns] = N.y;
                o[2 * ns] = D.x;
                o[3 * ns] = D.y;
                o[4 * ns] = (double)(S[u].E - S[u].EP);
            }
        };
        if (!SINGLE) keep(s_slot[jmax]);
        for (; i >= 0; --i) {
            step(i, std::true_type());
            if ((i & 3) == 0) rescale(true);
            if (!SINGLE && s_slot[i] >= 0) keep(s_slot[i]);
        }
#pragma unroll
        for (int u = 0; u < NM; ++u) {
            if (m[u] < 0) continue;
            const int ru = u == 0 || r == 0 ? r : g.nly - r;
            const int kyu = u == 0 ? ky : -ky;
            const double lyu = u == 0 ? ly : -ly;
            const double2 q0 = q0spec ? q0spec[(size_t)c * g.nly + ru] : make_double2(g.q0dc_fp, 0.0);
            double2 sh = make_double2(1.0, 0.0);
            if (g.do_shift) {
                const double th = lx * g.sx + lyu * g.sy;
                double sn, cs;
                sincos(th, &sn, &cs);
                sh = make_double2(cs, sn);
            }
            // q0 P / D_0
            const double2 D0 = make_double2(S[u].n[2], S[u].n[3]);
            const double dn = 1.0 / fma(D0.x, D0.x, D0.y * D0.y);
            const double2 G = dc_mul(q0, dc_mul(S[u].P, make_double2(D0.x * dn, -D0.y * dn)));
            const int e0 = S[u].EP - S[u].E;
            // the mirror of the mode, where it lies in the mode range
            const bool paired = -kx >= freq_min(g.nlx) && -kx <= freq_max(g.nlx) && -kyu >= freq_min(g.nly) &&
                                -kyu <= freq_max(g.nly);
            const int rm = paired ? index_of_freq(-kyu, g.nly) : 0;
            const int cm = paired ? index_of_freq(-kx, g.nlx) : 0;
            for (int s = 0; s < (SINGLE ? 1 : g.nsnap); ++s) {
                double2 N, D;
                int e = e0;
                if (SINGLE) {
                    N = make_double2(J[u].n[0], J[u].n[1]);
                    D = make_double2(J[u].n[2], J[u].n[3]);
                    e += J[u].E;
                } else {
                    const double *o = scratch + (size_t)s * 5 * ns + m[u];
                    N = make_double2(o[0], o[ns]);
                    D = make_double2(o[2 * ns], o[3 * ns]);
                    e += (int)o[4 * ns];
                }
                double2 q = dc_mul(D, G), p = dc_mul(N, G);
                q = make_double2(ldexp(q.x, e), ldexp(q.y, e));
                p = make_double2(ldexp(p.x, e), ldexp(p.y, e));
                if (g.precision == 0) {
                    p = round_c64(p);
                    q = round_c64(q);
                }
                if (g.do_shift) {
                    p = dc_mul(p, sh);
                    q = dc_mul(q, sh);
                }
                Xp[spec_idx(g, s, ru, c)] = p;
                Xq[spec_idx(g, s, ru, c)] = q;
                if (paired) {
                    Xp[spec_idx(g, s, rm, cm)] = make_double2(p.x, -p.y);
                    Xq[spec_idx(g, s, rm, cm)] = make_double2(q.x, -q.y);
                }
            }
        }
    }
}

// Launch of the FP64 sweeps.  The pipe passes one instruction per 16 clocks and
// SM, but of one warp only one per 64, so a launch takes (warps of the fullest
// SM, at least 4) x (instructions of a warp): one1 for a warp of single modes,
// one2 of pairs.  Pairs issue fewer in all but come in coarser units, and reach
// 95% of the pipe's rate (single modes 99%): 128^2 modes over 47 levels take 106
// us as singles, 191 us as pairs, 384^2 modes 885 and 821.  Up to some 9,000
// modes (fewer than two warps an SM) four lanes share a mode where the kernel
// has that form: lane4 instructions a lane.  One block per SM
// holds all its warps, at most 16: the number per SM is exact (small blocks are
// not dealt evenly), they share a level table, and more work goes in rounds of
// equal size, as a last round of fewer than four warps runs at their own rate.
// 512^2 modes over 207 levels: 3035 us in blocks of one warp, 2858 so (97% of
// the pipe for 14 warps an SM); the accurate sweep of 512^2 over 104: 869, 805.
struct Sweep64Launch {
    bool pairs, lanes;
    int threads;
    unsigned blocks;
};

static Sweep64Launch sweep64_launch(const SolveGeom &g, int nsm, double one1, double one2, double lane4 = 1e30)
{
    auto per_sm = [&](int64_t n) { return ((n + 31) / 32 + nsm - 1) / nsm; };
    auto units = [&](int64_t n) { return (double)std::max<int64_t>(per_sm(n), 4); };
    const int64_t n2 = sweep_items(g.nlx, g.nly).n;
    Sweep64Launch l;
    l.pairs = units(n2) * one2 < 0.95 * units(g.nsolved) * one1;
    l.lanes = units(4 * g.nsolved) * lane4 < 0.95 * std::min(units(n2) * one2, units(g.nsolved) * one1);
    const int64_t n = l.lanes ? 4 * g.nsolved : l.pairs ? n2 : g.nsolved, w = per_sm(n);
    const int64_t rounds = (w + SWEEP64_THREADS / 32 - 1) / (SWEEP64_THREADS / 32);
    l.threads = 32 * (int)((w + rounds - 1) / rounds);
    l.blocks = (unsigned)std::min<int64_t>((n + 31) / 32, nsm);
    return l;
}

cudaError_t launch_riccati64(const SolveGeom &g, const double *lvtab, const int *slot, const uint32_t *modes,
                             const double2 *q0spec, double *scratch, double2 *Xp, double2 *Xq, int nsm, cudaStream_t st)
{
    if (g.nsnap < 1 || g.nsolved == 0) return cudaSuccess;
    const size_t smem = (size_t)(g.nz - 1) * RT_N * sizeof(double) + (size_t)g.nz * sizeof(int) + 16;
    const double above = g.nz - 1 - g.jmax, below = g.jmax;
    const Sweep64Launch l = sweep64_launch(g, nsm, above * 30 + below * 40, above * 54 + below * 73);
    auto run = [&](auto k) { k<<<l.blocks, l.threads, smem, st>>>(g, lvtab, slot, modes, q0spec, scratch, Xp, Xq); };
    if (g.nsnap == 1)
        l.pairs ? run(riccati64_kernel<true, 2>) : run(riccati64_kernel<true, 1>);
    else
        l.pairs ? run(riccati64_kernel<false, 2>) : run(riccati64_kernel<false, 1>);
    return LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// FFT passes
// ---------------------------------------------------------------------------
// fwd_rows: lines are source rows y < ny, length nxe, input at offset px.
// Output A[c][y] (c < nlx truncated columns) scaled by 1/nxe.  smem: two
// ping-pong buffers of rows_per_cta lines, then the twiddles.
template <typename R>
__device__ __forceinline__ void fwd_row_lines(const SolveGeom &g, const FftPlan &pl,
                                              const typename cvec<R>::T *__restrict__ tw,
                                              const double *__restrict__ src, typename cvec<R>::T *__restrict__ A,
                                              int y0, int rows_per_cta, typename cvec<R>::T *smem)
{
    typedef typename cvec<R>::T C;
    const int n = pl.n;
    C *bufA = smem;
    C *bufB = bufA + (size_t)rows_per_cta * n;
    C *stw = bufB + (size_t)rows_per_cta * n;
    const int nl = min(rows_per_cta, g.ny - y0);
    for (int i = threadIdx.x; i < n; i += blockDim.x) stw[i] = tw[i];
    for (int i = threadIdx.x; i < nl * n; i += blockDim.x) {
        const int l = i / n, x = i - l * n;
        const int xs = x - g.px;
        R v = (xs >= 0 && xs < g.nx) ? (R)src[(size_t)(y0 + l) * g.nx + xs] : (R)0;
        bufA[i] = cx_make<C>(v, 0.0);
    }
    const int fx = freq_min(g.nlx);
    C *res = fft_run<C>(bufA, bufB, pl, nl, stw, -1, fx < 0 ? fx + n : fx, g.nlx);
    const R sc = (R)g.inv_nxe;
    for (int i = threadIdx.x; i < nl * g.nlx; i += blockDim.x) {
        const int c = i / nl, l = i - c * nl;
        const int kx = freq_of_index(c, g.nlx);
        const int pos = kx >= 0 ? kx : kx + n;
        C v = res[(size_t)l * n + pos];
        v.x *= sc;
        v.y *= sc;
        A[(size_t)c * g.ny + y0 + l] = v;
    }
}

// fwd_cols: lines are truncated columns c < nlx, length nye, input A[c][y] at
// offset py.  Output Q0[c][r] (r < nly) scaled by 1/nye.
template <typename R>
__device__ __forceinline__ void fwd_col_lines(const SolveGeom &g, const FftPlan &pl,
                                              const typename cvec<R>::T *__restrict__ tw,
                                              const typename cvec<R>::T *__restrict__ A,
                                              typename cvec<R>::T *__restrict__ Q0, int c0, int cols_per_cta,
                                              typename cvec<R>::T *smem)
{
    typedef typename cvec<R>::T C;
    const int n = pl.n;
    C *bufA = smem;
    C *bufB = bufA + (size_t)cols_per_cta * n;
    C *stw = bufB + (size_t)cols_per_cta * n;
    const int nl = min(cols_per_cta, g.nlx - c0);
    for (int i = threadIdx.x; i < n; i += blockDim.x) stw[i] = tw[i];
    for (int i = threadIdx.x; i < nl * n; i += blockDim.x) {
        const int l = i / n, y = i - l * n;
        const int ys = y - g.py;
        bufA[i] = (ys >= 0 && ys < g.ny) ? A[(size_t)(c0 + l) * g.ny + ys] : cx_make<C>(0.0, 0.0);
    }
    const int fy = freq_min(g.nly);
    C *res = fft_run<C>(bufA, bufB, pl, nl, stw, -1, fy < 0 ? fy + n : fy, g.nly);
    const R sc = (R)g.inv_nye;
    for (int i = threadIdx.x; i < nl * g.nly; i += blockDim.x) {
        const int l = i / g.nly, r = i - l * g.nly;
        const int ky = freq_of_index(r, g.nly);
        const int pos = ky >= 0 ? ky : ky + n;
        C v = res[(size_t)l * n + pos];
        v.x *= sc;
        v.y *= sc;
        Q0[(size_t)(c0 + l) * g.nly + r] = v;
    }
}

template <typename R>
__global__ void __launch_bounds__(256) fwd_rows_kernel(SolveGeom g, FftPlan pl, const typename cvec<R>::T *__restrict__ tw,
                                                       const double *__restrict__ src, typename cvec<R>::T *__restrict__ A,
                                                       int rows_per_cta)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    fwd_row_lines<R>(g, pl, tw, src, A, blockIdx.x * rows_per_cta, rows_per_cta, (typename cvec<R>::T *)smem_raw);
}

template <typename R>
__global__ void __launch_bounds__(256) fwd_cols_kernel(SolveGeom g, FftPlan pl, const typename cvec<R>::T *__restrict__ tw,
                                                       const typename cvec<R>::T *__restrict__ A,
                                                       typename cvec<R>::T *__restrict__ Q0, int cols_per_cta)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    fwd_col_lines<R>(g, pl, tw, A, Q0, blockIdx.x * cols_per_cta, cols_per_cta, (typename cvec<R>::T *)smem_raw);
}

// The forward passes of a batch's dispersion cases, blockIdx.y = case: one
// launch per pass (per-case launches of some 30 blocks each, one after
// another, left most of the device idle: 136 us for four 256 x 192 sources,
// 26 us so).
__device__ __forceinline__ void load_fwd_case(FwdCase *dst, const FwdCase *src)
{
    const int *s = (const int *)src;
    int *d = (int *)dst;
    for (int i = threadIdx.x; i < (int)(sizeof(FwdCase) / 4); i += blockDim.x) d[i] = s[i];
    __syncthreads();
}

__global__ void __launch_bounds__(256) fwd_rows_batch_kernel(const FwdCase *__restrict__ cases)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) FwdCase fc;
    if ((int)blockIdx.x * cases[blockIdx.y].rpc >= cases[blockIdx.y].g.ny) return;
    load_fwd_case(&fc, cases + blockIdx.y);
    fwd_row_lines<float>(fc.g, fc.plx, fc.twx, fc.src, fc.A, blockIdx.x * fc.rpc, fc.rpc, (float2 *)smem_raw);
}

__global__ void __launch_bounds__(256) fwd_cols_batch_kernel(const FwdCase *__restrict__ cases)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) FwdCase fc;
    if ((int)blockIdx.x * cases[blockIdx.y].cpc >= cases[blockIdx.y].g.nlx) return;
    load_fwd_case(&fc, cases + blockIdx.y);
    fwd_col_lines<float>(fc.g, fc.ply, fc.twy, fc.A, fc.Q0, blockIdx.x * fc.cpc, fc.cpc, (float2 *)smem_raw);
}

// out_cols: cols_per_cta band columns per CTA (blockIdx.x), one level (blockIdx.y).
template <typename R>
__global__ void __launch_bounds__(256) out_cols_kernel(SolveGeom g, FftPlan pl, const typename cvec<R>::T *__restrict__ tw,
                                                       const int4 *__restrict__ xband,
                                                       const typename cvec<R>::T *__restrict__ Xp,
                                                       const typename cvec<R>::T *__restrict__ Xq,
                                                       const double2 *__restrict__ dc,
                                                       typename cvec<R>::T *__restrict__ Cout, int cols_per_cta,
                                                       int *err)
{
    typedef typename cvec<R>::T C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if constexpr (sizeof(R) == 4) {
        // FP32 spectra are Hermitian-complete: the staged gather
        __shared__ uint64_t bar;
        if (threadIdx.x == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(&bar)),
                         "r"(1)
                         : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncthreads();
        if (!out_col_lines_staged(g, pl, tw, xband, Xp, Xq, dc, Cout, blockIdx.x * cols_per_cta, cols_per_cta,
                                  blockIdx.y, (C *)smem_raw, &bar) &&
            threadIdx.x == 0 && err)
            atomicExch(err, BLDFM_ERR_TIMEOUT_DEV);
    } else {
        out_col_lines<R>(g, pl, tw, xband, Xp, Xq, dc, Cout, blockIdx.x * cols_per_cta, cols_per_cta, blockIdx.y,
                         (C *)smem_raw);
    }
}

// out_rows: rows_per_cta output rows per CTA, one level (blockIdx.y).
template <typename R>
__global__ void __launch_bounds__(256) out_rows_kernel(SolveGeom g, FftPlan pl, const typename cvec<R>::T *__restrict__ tw,
                                                       const int4 *__restrict__ xband,
                                                       const typename cvec<R>::T *__restrict__ Cin,
                                                       double *__restrict__ conc, double *__restrict__ flx,
                                                       int rows_per_cta, int *err)
{
    typedef typename cvec<R>::T C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    out_row_lines<R>(g, pl, tw, xband, Cin, conc, flx, blockIdx.x * rows_per_cta, rows_per_cta, blockIdx.y,
                     (C *)smem_raw, err);
}

// ---------------------------------------------------------------------------
// small utility kernels
// ---------------------------------------------------------------------------
// twiddle table tw[m] = exp(-2 pi i m / n) converted from the FP64 table
__global__ void tw_to_float_kernel(const double2 *__restrict__ src, float2 *__restrict__ dst, int n)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = make_float2((float)src[i].x, (float)src[i].y);
}

__global__ void spec_to_float_kernel(const double2 *__restrict__ src, float2 *__restrict__ dst, int64_t n)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = make_float2((float)src[i].x, (float)src[i].y);
}

// non-finite detector over the outputs
__global__ void nonfinite_kernel(const double *__restrict__ a, const double *__restrict__ b, int64_t n, int *flag)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (!isfinite(a[i]) || !isfinite(b[i])) {
            atomicExch(flag, 1);
            return;
        }
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------


cudaError_t launch_sweep64(const SolveGeom &g, const double *lvtab, const int *slot, const uint32_t *modes,
                           const double2 *q0spec, double2 *snap, double2 *top, int *err, int nsm, cudaStream_t st)
{
    const int L = g.nz - 1;
    const size_t smem = (size_t)L * BLDFM_LV64 * sizeof(double) + (size_t)g.nz * sizeof(int) + 16;
    static uint64_t attr = 0;
    if (first_on_device(attr)) {
        cudaFuncSetAttribute(sweep64_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(sweep64_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(sweep64_lanes_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    }
    const Sweep64Launch l = sweep64_launch(g, nsm, 68, 124, 33);
    if (l.lanes)
        sweep64_lanes_kernel<<<l.blocks, l.threads, smem, st>>>(g, lvtab, slot, modes, q0spec, snap, top, err);
    else if (l.pairs)
        sweep64_kernel<2><<<l.blocks, l.threads, smem, st>>>(g, lvtab, slot, modes, q0spec, snap, top, err);
    else
        sweep64_kernel<1><<<l.blocks, l.threads, smem, st>>>(g, lvtab, slot, modes, q0spec, snap, top, err);
    return LAUNCH_CHECK();
}

cudaError_t launch_combine64(const SolveGeom &g, const uint32_t *modes, const double2 *eig, const double2 *snap,
                             const double2 *top, double2 *Xp, double2 *Xq, cudaStream_t st)
{
    if (g.nsolved == 0) return cudaSuccess;
    // small blocks: a thread's work is a serial chain per level, and few modes
    // in large ones leave SMs idle (14,250 modes, nine levels: 23 us in blocks
    // of 256, 17 so; 4,096 modes and one level: 11, 6)
    const int threads = 64;
    const unsigned blocks = (unsigned)((g.nsolved + threads - 1) / threads);
    combine64_kernel<<<blocks, threads, 0, st>>>(g, modes, eig, snap, top, Xp, Xq);
    return LAUNCH_CHECK();
}

cudaError_t launch_trapezoid64(const SolveGeom &g, const double *lvtab, const int *slot, const double2 *q0spec,
                               double p000, double2 *dc, cudaStream_t st)
{
    const size_t smem = (size_t)(g.nz > 1 ? g.nz - 1 : 1) * sizeof(double2) + (size_t)g.nz * sizeof(int);
    trapezoid_kernel<double2><<<1, 256, smem, st>>>(g, lvtab, slot, q0spec, p000, dc, nullptr);
    return LAUNCH_CHECK();
}

// FP64 partial sums of the source field: CTA b of DC_PARTS sums its slice in a
// fixed order (deterministic), thread sums then a shared-memory tree
__device__ __forceinline__ void dc_partial_sum(const double *__restrict__ src, int64_t n, double *__restrict__ dcp)
{
    __shared__ double red[256];
    const int64_t chunk = (n + DC_PARTS - 1) / DC_PARTS;
    const int64_t b0 = (int64_t)blockIdx.x * chunk, b1 = b0 + chunk < n ? b0 + chunk : n;
    double acc = 0.0;
    for (int64_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) acc += src[i];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) dcp[blockIdx.x] = red[0];
}

__global__ void __launch_bounds__(256) dc_partial_kernel(const double *__restrict__ src, int64_t n,
                                                         double *__restrict__ dcp)
{
    dc_partial_sum(src, n, dcp);
}

__global__ void __launch_bounds__(256) dc_partial_batch_kernel(const FwdCase *__restrict__ cases)
{
    const FwdCase &c = cases[blockIdx.y];
    dc_partial_sum(c.src, (int64_t)c.g.nx * c.g.ny, c.dcp);
}

cudaError_t launch_trapezoid32(const SolveGeom &g, const double *lvtab, const int *slot, const float2 *q0spec,
                               double p000, double2 *dc, cudaStream_t st, const double *src, double *dcp)
{
    const size_t smem = (size_t)(g.nz > 1 ? g.nz - 1 : 1) * sizeof(double2) + (size_t)g.nz * sizeof(int);
    const bool exact = src && dcp;
    if (exact) dc_partial_kernel<<<DC_PARTS, 256, 0, st>>>(src, (int64_t)g.nx * g.ny, dcp);
    trapezoid_kernel<float2><<<1, 256, smem, st>>>(g, lvtab, slot, q0spec, p000, dc, exact ? dcp : nullptr);
    return LAUNCH_CHECK();
}

cudaError_t launch_analytic64(const SolveGeom &g, const uint32_t *modes, const double2 *eig, const double2 *q0spec,
                              double p000, double kzinv, double hlev, double2 *Xp, double2 *Xq, double2 *dc,
                              cudaStream_t st)
{
    if (g.nsolved > 0) {
        const int threads = 256;
        const unsigned blocks = (unsigned)((g.nsolved + threads - 1) / threads);
        analytic64_kernel<<<blocks, threads, 0, st>>>(g, modes, eig, q0spec, kzinv, hlev, Xp, Xq);
    }
    if (q0spec) analytic_dc_kernel<<<1, 32, 0, st>>>(g, q0spec, p000, kzinv, hlev, dc);
    return LAUNCH_CHECK();
}

cudaError_t launch_riccati32(const SolveGeom &g, const float *lv32, const int *slot, const uint32_t *modes,
                             const float2 *q0spec, float *scratch, float2 *Xp, float2 *Xq, float ax, float ay,
                             int *err, int nsm, int threads, cudaStream_t st)
{
    const int L = g.nz - 1;
    const size_t smem = (size_t)L * BLDFM_LV32 * sizeof(float) + (size_t)g.nz * sizeof(int) + 16;
    static uint64_t attr = 0;
    if (first_on_device(attr)) {
        cudaFuncSetAttribute(riccati32_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(riccati32_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(riccati32_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(riccati32_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    }
    if (threads <= 0) threads = 256;
    const int64_t per_thread = g.nsnap == 1 ? 2 : 1;  // modes per thread
    int64_t blocks = (g.nsolved + per_thread * threads - 1) / (per_thread * threads);
    if (blocks < 1) blocks = 1;
    if (blocks > 64LL * nsm) blocks = 64LL * nsm;
    const bool single = g.nsnap == 1;
    if (g.nsnap < 1) return cudaSuccess;  // no output level inside the grid: spectra stay zero
    if (g.iso) {
        if (single)
            riccati32_kernel<true, true><<<(unsigned)blocks, threads, smem, st>>>(g, lv32, slot, modes, q0spec, scratch,
                                                                                Xp, Xq, ax, ay, err);
        else
            riccati32_kernel<true, false><<<(unsigned)blocks, threads, smem, st>>>(g, lv32, slot, modes, q0spec,
                                                                                 scratch, Xp, Xq, ax, ay, err);
    } else {
        if (single)
            riccati32_kernel<false, true><<<(unsigned)blocks, threads, smem, st>>>(g, lv32, slot, modes, q0spec,
                                                                                 scratch, Xp, Xq, ax, ay, err);
        else
            riccati32_kernel<false, false><<<(unsigned)blocks, threads, smem, st>>>(g, lv32, slot, modes, q0spec,
                                                                                  scratch, Xp, Xq, ax, ay, err);
    }
    return LAUNCH_CHECK();
}

static int device_sms()
{
    int dev = 0, nsm = 152;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}

// Lines of a forward pass per block: as many as fit about 96 KB, at most 8,
// but at least two blocks per SM over the launch (a single source has few
// lines: the two passes of 190 x 150 in FP64 took 136 us at up to eight lines a
// block, 52 us so).
int fwd_lines_per_cta(int n, size_t elem, int lines, int nsm)
{
    int l = (int)((96 * 1024) / (2 * (size_t)n * elem));
    l = std::min(std::max(l, 1), 8);
    while (l > 1 && (lines + l - 1) / l < 2 * nsm) --l;
    return l;
}

size_t fwd_smem(int n, size_t elem, int lines) { return (2 * (size_t)lines + 1) * n * elem; }

template <typename R>
static void set_fft_smem_attr()
{
    static uint64_t done = 0;
    if (!first_on_device(done)) return;
    cudaFuncSetAttribute(fwd_rows_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(fwd_cols_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(out_cols_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(out_rows_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (sizeof(R) == 4) {
        cudaFuncSetAttribute(fwd_rows_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(fwd_cols_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    }
}

template <typename R>
cudaError_t launch_forward_fft(const SolveGeom &g, const FftPlan &plx, const FftPlan &ply,
                               const typename cvec<R>::T *twx, const typename cvec<R>::T *twy, const double *src,
                               typename cvec<R>::T *A, typename cvec<R>::T *Q0, cudaStream_t st)
{
    typedef typename cvec<R>::T C;
    set_fft_smem_attr<R>();
    if (g.ny <= 0 || g.nlx <= 0) return cudaSuccess;
    const int nsm = device_sms();
    const int rpc = fwd_lines_per_cta(plx.n, sizeof(C), g.ny, nsm);
    fwd_rows_kernel<R><<<(g.ny + rpc - 1) / rpc, 256, fwd_smem(plx.n, sizeof(C), rpc), st>>>(g, plx, twx, src, A, rpc);
    const int cpc = fwd_lines_per_cta(ply.n, sizeof(C), g.nlx, nsm);
    fwd_cols_kernel<R><<<(g.nlx + cpc - 1) / cpc, 256, fwd_smem(ply.n, sizeof(C), cpc), st>>>(g, ply, twy, A, Q0, cpc);
    return LAUNCH_CHECK();
}

template <typename R>
cudaError_t launch_output_fft(const SolveGeom &g, const FftPlan &plx, const FftPlan &ply,
                              const typename cvec<R>::T *twx, const typename cvec<R>::T *twy, const int4 *xband,
                              const typename cvec<R>::T *Xp, const typename cvec<R>::T *Xq, const double2 *dc,
                              typename cvec<R>::T *Cbuf, double *conc, double *flx, int *err, cudaStream_t st)
{
    typedef typename cvec<R>::T C;
    set_fft_smem_attr<R>();
    if (g.nbx <= 0 || g.out_ny <= 0 || g.out_nx <= 0 || g.nlvls <= 0) return cudaSuccess;
    // lines per CTA: as many as shared memory allows, but at least two CTAs
    // per SM over the launch (a single footprint has few lines)
    const int nsm = device_sms();
    int cpc = out_cols_per_cta(ply.n, sizeof(C));
    while (cpc > 1 && (int64_t)((g.nbx + cpc - 1) / cpc) * g.nlvls < 2 * (int64_t)nsm) cpc >>= 1;
    dim3 gc((g.nbx + cpc - 1) / cpc, g.nlvls);
    out_cols_kernel<R><<<gc, 256, (2 * (size_t)cpc + 1) * ply.n * sizeof(C), st>>>(g, ply, twy, xband, Xp, Xq, dc,
                                                                                   Cbuf, cpc, err);
    // two rows per CTA in FP32, one in FP64, bounded by shared memory and by
    // the same two CTAs per SM
    int rpc = sizeof(C) == 8 ? 2 : 1;
    while (rpc > 1 && (2 * (size_t)rpc + 1) * plx.n * sizeof(C) > 190 * 1024) --rpc;
    while (rpc > 1 && (int64_t)((g.out_ny + rpc - 1) / rpc) * g.nlvls < 2 * (int64_t)nsm) --rpc;
    dim3 gr((g.out_ny + rpc - 1) / rpc, g.nlvls);
    out_rows_kernel<R><<<gr, 256, (2 * (size_t)rpc + 1) * plx.n * sizeof(C), st>>>(g, plx, twx, xband, Cbuf, conc,
                                                                                   flx, rpc, err);
    return LAUNCH_CHECK();
}

static const int FWD_MAX_CASES = 65535;  // the grid's y limit

cudaError_t launch_forward_batch(const FwdCase *cases, int n, int rows, size_t row_smem, int cols, size_t col_smem,
                                 cudaStream_t st)
{
    set_fft_smem_attr<float>();
    for (int i = 0; i < n; i += FWD_MAX_CASES) {
        const int m = n - i < FWD_MAX_CASES ? n - i : FWD_MAX_CASES;
        fwd_rows_batch_kernel<<<dim3(rows, m), 256, row_smem, st>>>(cases + i);
        fwd_cols_batch_kernel<<<dim3(cols, m), 256, col_smem, st>>>(cases + i);
    }
    return LAUNCH_CHECK();
}

cudaError_t launch_dc_batch(const FwdCase *cases, int n, int max_nz, cudaStream_t st)
{
    set_fft_smem_attr<float>();
    for (int i = 0; i < n; i += FWD_MAX_CASES)
        dc_partial_batch_kernel<<<dim3(DC_PARTS, n - i < FWD_MAX_CASES ? n - i : FWD_MAX_CASES), 256, 0, st>>>(cases +
                                                                                                              i);
    const size_t smem = (size_t)(max_nz > 1 ? max_nz - 1 : 1) * sizeof(double2) + (size_t)max_nz * sizeof(int);
    trapezoid_batch_kernel<<<n, 256, smem, st>>>(cases);
    return LAUNCH_CHECK();
}

template cudaError_t launch_forward_fft<double>(const SolveGeom &, const FftPlan &, const FftPlan &, const double2 *,
                                                const double2 *, const double *, double2 *, double2 *, cudaStream_t);
template cudaError_t launch_forward_fft<float>(const SolveGeom &, const FftPlan &, const FftPlan &, const float2 *,
                                               const float2 *, const double *, float2 *, float2 *, cudaStream_t);
template cudaError_t launch_output_fft<double>(const SolveGeom &, const FftPlan &, const FftPlan &, const double2 *,
                                               const double2 *, const int4 *, const double2 *, const double2 *,
                                               const double2 *, double2 *, double *, double *, int *, cudaStream_t);
template cudaError_t launch_output_fft<float>(const SolveGeom &, const FftPlan &, const FftPlan &, const float2 *,
                                              const float2 *, const int4 *, const float2 *, const float2 *,
                                              const double2 *, float2 *, double *, double *, int *, cudaStream_t);

cudaError_t launch_tw_to_float(const double2 *src, float2 *dst, int n, cudaStream_t st)
{
    tw_to_float_kernel<<<(n + 255) / 256, 256, 0, st>>>(src, dst, n);
    return LAUNCH_CHECK();
}

cudaError_t launch_spec_to_float(const double2 *src, float2 *dst, int64_t n, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    spec_to_float_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(src, dst, n);
    return LAUNCH_CHECK();
}

cudaError_t launch_nonfinite(const double *a, const double *b, int64_t n, int *flag, int nsm, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    int64_t blocks = (n + 255) / 256;
    if (blocks > 4LL * nsm) blocks = 4LL * nsm;
    nonfinite_kernel<<<(unsigned)blocks, 256, 0, st>>>(a, b, n, flag);
    return LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// FMA throughput probe: independent FMA chains per thread, CUDA-event timed.
// Measures the FP32 / FP64 pipe peaks that bound the sweep kernels.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) fma_peak_kernel(T *out, int iters, T b, T c)
{
    T a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = (T)(threadIdx.x + k) * (T)1e-3;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = fma(a[k], b, c);
    }
    T s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += a[k];
    if (s == (T)-12345.678) out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

// Packed FP32: eight independent f32x2 FMA chains per thread.
__global__ void __launch_bounds__(256) fma2_peak_kernel(float *out, int iters, float b, float c)
{
    float2 a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = make_float2((float)(threadIdx.x + k) * 1e-3f, (float)(threadIdx.x + 2 * k) * 1e-3f);
    const float2 b2 = make_float2(b, b), c2 = make_float2(c, c);
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = __ffma2_rn(a[k], b2, c2);
    }
    float s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += a[k].x + a[k].y;
    if (s == -12345.678f) out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

cudaError_t run_fma_peak(int kind, int nsm, cudaStream_t st, double *flops_per_s)
{
    const bool fp64 = kind == 1;
    const int threads = 256, blocks = nsm * 8;
    const int iters = fp64 ? 2048 : (kind == 2 ? 32768 : 65536);
    void *out = nullptr;
    cudaError_t e = cudaMalloc(&out, (size_t)threads * blocks * 8);
    if (e != cudaSuccess) return e;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    float best = 1e30f;
    for (int rep = 0; rep < 4; ++rep) {
        cudaEventRecord(a, st);
        if (fp64)
            fma_peak_kernel<double><<<blocks, threads, 0, st>>>((double *)out, iters, 0.999999, 1e-7);
        else if (kind == 2)
            fma2_peak_kernel<<<blocks, threads, 0, st>>>((float *)out, iters, 0.999999f, 1e-7f);
        else
            fma_peak_kernel<float><<<blocks, threads, 0, st>>>((float *)out, iters, 0.999999f, 1e-7f);
        cudaEventRecord(b, st);
        cudaEventSynchronize(b);
        float ms = 0;
        cudaEventElapsedTime(&ms, a, b);
        if (rep > 0 && ms < best) best = ms;
    }
    e = cudaGetLastError();
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(out);
    *flops_per_s = 2.0 * 8.0 * (kind == 2 ? 2 : 1) * iters * (double)threads * blocks / (best * 1e-3);
    return e;
}

// Shared-memory limits of every kernel, set once per device before any launch
// (and so before any stream capture).
void prepare_kernel_attributes()
{
    set_fft_smem_attr<double>();
    set_fft_smem_attr<float>();
    cudaFuncSetAttribute(sweep64_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(sweep64_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(riccati64_kernel<true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, RICC64_SMEM);
    cudaFuncSetAttribute(riccati64_kernel<true, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, RICC64_SMEM);
    cudaFuncSetAttribute(riccati64_kernel<false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, RICC64_SMEM);
    cudaFuncSetAttribute(riccati64_kernel<false, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, RICC64_SMEM);
    cudaFuncSetAttribute(riccati32_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(riccati32_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(riccati32_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(riccati32_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
}
