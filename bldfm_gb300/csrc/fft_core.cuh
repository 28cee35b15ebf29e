// Mixed-radix Stockham autosort FFT on lines held in shared memory.
//
// State after stage q (radix p, L_q = L_{q-1} * p, r_q = N / L_q):
//   y_q[j, k] = sum_{n < L_q} x[n r_q + k] w_{L_q}^{j n},  stored at j*r_q + k.
// One butterfly per (j1 < L_{q-1}, k < r_q):
//   y_q[j1 + L_{q-1} j2, k] = sum_t (w_N^{j1 t r_q} y_{q-1}[j1, t r_q + k]) w_p^{j2 t}.
// Input and output are in natural order (autosort), ping-ponging between two
// buffers.  Twiddles come from a table tw[m] = exp(-2 pi i m / N); the
// inverse sign conjugates them.
#pragma once

#include "common.h"


template <typename C>
__device__ __forceinline__ C cx_make(double a, double b)
{
    C o;
    o.x = a;
    o.y = b;
    return o;
}

template <typename C>
__device__ __forceinline__ C cx_mul(C a, C b)
{
    C o;
    o.x = a.x * b.x - a.y * b.y;
    o.y = a.x * b.y + a.y * b.x;
    return o;
}

template <typename C>
__device__ __forceinline__ C cx_add(C a, C b)
{
    C o;
    o.x = a.x + b.x;
    o.y = a.y + b.y;
    return o;
}

template <typename C>
__device__ __forceinline__ C cx_sub(C a, C b)
{
    C o;
    o.x = a.x - b.x;
    o.y = a.y - b.y;
    return o;
}

// multiply by -i*sign... helper: rotate by +/- 90 degrees: (x + iy) * (i*s) = (-s y, s x)
template <typename C>
__device__ __forceinline__ C cx_rot(C a, float s)
{
    C o;
    o.x = -s * a.y;
    o.y = s * a.x;
    return o;
}

template <typename C, int SIGN>
__device__ __forceinline__ C tw_get(const C *tw, int m)
{
    C w = tw[m];
    if (SIGN > 0) w.y = -w.y;
    return w;
}

__device__ __forceinline__ uint32_t fdiv(uint32_t x, const FDiv &f)
{
    return f.s < 0 ? x : (__umulhi(x, f.m) >> f.s);
}

// Radix-p butterfly body for one (j1, k).  u[] already twiddled.
template <typename C, int P, int SIGN>
__device__ __forceinline__ void dft_small(C *u, const C *tw, int n)
{
    constexpr int sign = SIGN;
    typedef decltype(u[0].x) RR;
    if (P == 2) {
        C a = u[0], b = u[1];
        u[0] = cx_add(a, b);
        u[1] = cx_sub(a, b);
    } else if (P == 4) {
        C a0 = cx_add(u[0], u[2]), a1 = cx_sub(u[0], u[2]);
        C b0 = cx_add(u[1], u[3]), b1 = cx_sub(u[1], u[3]);
        // w_4 = exp(sign * 2 pi i / 4) = sign*i  (forward sign = -1 -> -i)
        C b1r = cx_rot(b1, (float)sign);
        u[0] = cx_add(a0, b0);
        u[2] = cx_sub(a0, b0);
        u[1] = cx_add(a1, b1r);
        u[3] = cx_sub(a1, b1r);
    } else if (P == 3) {
        // w_3 = -1/2 + sign * i sqrt(3)/2
        const RR c1 = (RR)-0.5;
        const RR s1 = (RR)(sign * 0.86602540378443864676372317075294);
        C s = cx_add(u[1], u[2]);
        C d = cx_sub(u[1], u[2]);
        C a = u[0];
        u[0] = cx_add(a, s);
        C m;
        m.x = a.x + c1 * s.x;
        m.y = a.y + c1 * s.y;
        C r;  // i * s1 * d
        r.x = -s1 * d.y;
        r.y = s1 * d.x;
        u[1] = cx_add(m, r);
        u[2] = cx_sub(m, r);
    } else if (P == 8) {
        // two radix-4 layers with internal twiddles w_8^{k}
        C a[4], b[4];
        for (int t = 0; t < 4; ++t) {
            a[t] = u[2 * t];
            b[t] = u[2 * t + 1];
        }
        // radix-4 on even and odd halves
        {
            C x0 = cx_add(a[0], a[2]), x1 = cx_sub(a[0], a[2]);
            C y0 = cx_add(a[1], a[3]), y1 = cx_rot(cx_sub(a[1], a[3]), (float)sign);
            a[0] = cx_add(x0, y0);
            a[2] = cx_sub(x0, y0);
            a[1] = cx_add(x1, y1);
            a[3] = cx_sub(x1, y1);
        }
        {
            C x0 = cx_add(b[0], b[2]), x1 = cx_sub(b[0], b[2]);
            C y0 = cx_add(b[1], b[3]), y1 = cx_rot(cx_sub(b[1], b[3]), (float)sign);
            b[0] = cx_add(x0, y0);
            b[2] = cx_sub(x0, y0);
            b[1] = cx_add(x1, y1);
            b[3] = cx_sub(x1, y1);
        }
        const RR h = (RR)0.70710678118654752440084436210485;
        // b[k] *= w_8^k, w_8 = (1 + sign*i)/sqrt2
        C t1;
        t1.x = h * (b[1].x - sign * b[1].y);
        t1.y = h * (b[1].y + sign * b[1].x);
        b[1] = t1;
        b[2] = cx_rot(b[2], (float)sign);
        C t3;  // w_8^3 = (-1 + sign*i)/sqrt2
        t3.x = h * (-b[3].x - sign * b[3].y);
        t3.y = h * (-b[3].y + sign * b[3].x);
        b[3] = t3;
        for (int t = 0; t < 4; ++t) {
            u[t] = cx_add(a[t], b[t]);
            u[t + 4] = cx_sub(a[t], b[t]);
        }
    } else if (P == 5 && sizeof(RR) == 8) {
        // FP64: symmetric inputs folded (36 operations where the direct sums,
        // whose order FP32 keeps, take 104)
        const RR c1 = (RR)0.30901699437494742410229341718282, c2 = (RR)-0.80901699437494742410229341718282;
        const RR s1 = (RR)(sign * 0.95105651629515357211643933337938), s2 = (RR)(sign * 0.58778525229247312916870595463907);
        const C S1 = cx_add(u[1], u[4]), D1 = cx_sub(u[1], u[4]), S2 = cx_add(u[2], u[3]), D2 = cx_sub(u[2], u[3]);
        const C a = u[0];
        C A1, A2, B1, B2;
        A1.x = fma(c2, S2.x, fma(c1, S1.x, a.x));
        A1.y = fma(c2, S2.y, fma(c1, S1.y, a.y));
        A2.x = fma(c1, S2.x, fma(c2, S1.x, a.x));
        A2.y = fma(c1, S2.y, fma(c2, S1.y, a.y));
        B1.x = fma(s2, D2.x, s1 * D1.x);
        B1.y = fma(s2, D2.y, s1 * D1.y);
        B2.x = fma(-s1, D2.x, s2 * D1.x);
        B2.y = fma(-s1, D2.y, s2 * D1.y);
        u[0] = cx_add(a, cx_add(S1, S2));
        B1 = cx_rot(B1, 1.f);  // i B
        B2 = cx_rot(B2, 1.f);
        u[1] = cx_add(A1, B1);
        u[4] = cx_sub(A1, B1);
        u[2] = cx_add(A2, B2);
        u[3] = cx_sub(A2, B2);
    } else if (P == 5) {
        C o[5];
        for (int j = 0; j < 5; ++j) {
            C acc = u[0];
            for (int t = 1; t < 5; ++t) {
                int m = ((j * t) % 5) * (n / 5);
                acc = cx_add(acc, cx_mul(u[t], tw_get<C, SIGN>(tw, m)));
            }
            o[j] = acc;
        }
        for (int j = 0; j < 5; ++j) u[j] = o[j];
    }
}

// One Stockham stage of specialised radix P over nlines lines of length n;
// stage constants from the plan (rq, divisions by rq and by n / P).
template <typename C, int P, int SIGN>
__device__ void stage_p(const C *__restrict__ src, C *__restrict__ dst, int n, int nlines, int L1, int rq,
                        const FDiv drq, const FDiv dnb, const C *__restrict__ tw)
{
    const int nb = n / P;  // butterflies per line
    const int total = nb * nlines;
    for (int b = threadIdx.x; b < total; b += blockDim.x) {
        const int line = (int)fdiv((uint32_t)b, dnb);
        const int loc = b - line * nb;
        const int j1 = (int)fdiv((uint32_t)loc, drq);
        const int k = loc - j1 * rq;
        const C *s = src + (size_t)line * n;
        C *d = dst + (size_t)line * n;
        C u[P];
        const int base = j1 * rq * P + k;
#pragma unroll
        for (int t = 0; t < P; ++t) {
            C v = s[base + t * rq];
            if (t > 0 && j1 > 0) v = cx_mul(v, tw_get<C, SIGN>(tw, j1 * t * rq));
            u[t] = v;
        }
        dft_small<C, P, SIGN>(u, tw, n);
#pragma unroll
        for (int t = 0; t < P; ++t) d[(j1 + L1 * t) * rq + k] = u[t];
    }
}

// Direct sums of a generic stage, inputs twiddled: outputs a .. a + m - 1 (mod
// p) of bl butterflies, U outputs of U butterflies per thread.
template <typename C, int SIGN, int U>
__device__ __forceinline__ void generic_sums(const C *__restrict__ src, C *__restrict__ dst, int n, int bl, int L1,
                                             int p, int rq, const FDiv drq, const FDiv dnb, const C *__restrict__ tw,
                                             int a, int m)
{
    const int nb = n / p, bh = (bl + U - 1) / U, mh = (m + U - 1) / U;
    for (int b = threadIdx.x; b < bh * mh; b += blockDim.x) {
        const int jh = b / bh, b0 = b - jh * bh;
        bool on_b[U], on_j[U];  // the last thread of an odd count repeats its first
        int j2[U], step[U], at[U], out[U];  // at: j2 t n / p mod n
        const C *s[U];
        C acc[U][U];
#pragma unroll
        for (int v = 0; v < U; ++v) {
            on_j[v] = U * jh + v < m;
            j2[v] = a + U * jh + (on_j[v] ? v : 0);
            if (j2[v] >= p) j2[v] -= p;
            step[v] = j2[v] * nb;
            at[v] = 0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            on_b[u] = b0 + u * bh < bl;
            const int bb = b0 + (on_b[u] ? u * bh : 0);
            const int line = (int)fdiv((uint32_t)bb, dnb);
            const int loc = bb - line * nb;
            const int j1 = (int)fdiv((uint32_t)loc, drq);
            const int k = loc - j1 * rq;
            s[u] = src + (size_t)line * n + j1 * rq * p + k;
            out[u] = line * n + j1 * rq + k;
#pragma unroll
            for (int v = 0; v < U; ++v) acc[u][v] = s[u][0];
        }
#pragma unroll (U == 1 ? 4 : 2)
        for (int t = 1; t < p; ++t) {
            C x[U], w[U];
#pragma unroll
            for (int v = 0; v < U; ++v) {
                at[v] += step[v];
                if (at[v] >= n) at[v] -= n;
                w[v] = tw_get<C, SIGN>(tw, at[v]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                s[u] += rq;
                x[u] = *s[u];
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int v = 0; v < U; ++v) acc[u][v] = cx_add(acc[u][v], cx_mul(x[u], w[v]));
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int v = 0; v < U; ++v)
                if (on_b[u] && on_j[v]) dst[out[u] + L1 * j2[v] * rq] = acc[u][v];
    }
}

// the one-by-one form, out of line: both forms inlined would raise the kernels'
// registers (the persistent row pass from 64 to 128)
template <typename C, int SIGN>
__device__ __noinline__ void generic_sums_1(const C *__restrict__ src, C *__restrict__ dst, int n, int bl, int L1,
                                            int p, int rq, const FDiv drq, const FDiv dnb, const C *__restrict__ tw,
                                            int a, int m)
{
    generic_sums<C, SIGN, 1>(src, dst, n, bl, L1, p, rq, drq, dnb, tw, a, m);
}

// Generic radix p (a prime >= 7, in practice a large factor of a ragged grid),
// O(p) work per output, every output its own thread's: a butterfly's p^2
// products are spread over the block (one thread per butterfly left 2 of 256
// threads busy on 386 = 2 x 193).  The inputs are twiddled in place first, so
// no output repeats that product.
//
// FP64 is bound by the FP64 pipe (2 lanes per clock and SM), so it folds the
// symmetric inputs, S_t = x_t + x_{p-t} and D_t = x_t - x_{p-t}, in place
// (S_t at t, D_t at p - t) and forms the outputs j and p - j together,
//   X_{j, p-j} = (x_0 + sum_t S_t cos(2 pi j t / p)) +/- i (sum_t D_t sin(2 pi j t / p)):
// a quarter of the direct sum's FMAs, and fewer roundings.  FP32 keeps the
// direct sum in its order.
//
// Only the outputs j2 = a .. a + m - 1 (mod p) are formed: all of them in an
// inner stage, in the last one (rq = 1, output j1 + L1 j2) those that hold the
// transform outputs the caller reads, the window of a solve with a halo or the
// kept band of a source.  The arc's pairs (j, p - j) are an arc again.  A third
// of each line is read where the halo is as wide as the grid: the FP64 solve
// 190 x 150 (570 = 30 x 19, 530 = 10 x 53) took 689 us with every output formed,
// 606 us so.
template <typename C, int SIGN>
__device__ void stage_generic(C *__restrict__ src, C *__restrict__ dst, int n, int nlines, int L1, int p, int rq,
                              const FDiv drq, const FDiv dnb, const C *__restrict__ tw, int a, int m)
{
    typedef decltype(src[0].x) RR;
    const int nb = n / p;
    const int np_ = n / p;
    if constexpr (sizeof(RR) == 8) {
        const int h = p >> 1, bl = nb * nlines;  // p is odd
        const int e = a + m - 1, ea = min(a, p - a), ee = e >= p ? min(e - p, 2 * p - e) : min(e, p - e);
        const bool all = m >= p;
        const int jmin = all || a == 0 || e >= p ? 0 : min(ea, ee);
        const int jmax = all || (a <= h + 1 && e >= h) || e >= h + p ? h : max(ea, ee);
        for (int b = threadIdx.x; b < bl * h; b += blockDim.x) {
            const int t = 1 + b / bl, bb = b - (t - 1) * bl;  // consecutive threads: consecutive butterflies
            const int line = (int)fdiv((uint32_t)bb, dnb);
            const int loc = bb - line * nb;
            const int j1 = (int)fdiv((uint32_t)loc, drq);
            C *s = src + (size_t)line * n + j1 * rq * p + (loc - j1 * rq);
            C x = s[t * rq], y = s[(p - t) * rq];
            if (j1 > 0) {
                x = cx_mul(x, tw_get<C, SIGN>(tw, j1 * t * rq));
                y = cx_mul(y, tw_get<C, SIGN>(tw, j1 * (p - t) * rq));
            }
            s[t * rq] = cx_add(x, y);
            s[(p - t) * rq] = cx_sub(x, y);
        }
        __syncthreads();
        for (int b = threadIdx.x; b < bl * (jmax - jmin + 1); b += blockDim.x) {
            const int j0 = b / bl, bb = b - j0 * bl, j = jmin + j0;
            const int line = (int)fdiv((uint32_t)bb, dnb);
            const int loc = bb - line * nb;
            const int j1 = (int)fdiv((uint32_t)loc, drq);
            const int k = loc - j1 * rq;
            const C *s = src + (size_t)line * n + j1 * rq * p + k;
            C *d = dst + (size_t)line * n + k;
            C A = s[0], B = cx_make<C>(0.0, 0.0);
            int jt = 0;  // j t mod p
            for (int t = 1; t <= h; ++t) {
                jt += j;
                if (jt >= p) jt -= p;
                const C w = tw[jt * np_];  // (cos, -sin)
                const C S = s[t * rq], D = s[(p - t) * rq];
                A.x = fma(S.x, w.x, A.x);
                A.y = fma(S.y, w.x, A.y);
                B.x = fma(D.x, w.y, B.x);
                B.y = fma(D.y, w.y, B.y);
            }
            // i SIGN (-B): the table holds -sin
            const C r = cx_rot(B, (float)-SIGN);
            d[(j1 + L1 * j) * rq] = cx_add(A, r);
            if (j > 0) d[(j1 + L1 * (p - j)) * rq] = cx_sub(A, r);
        }
    } else {
        const int bl = nb * nlines;
        if (L1 > 1) {
            for (int b = threadIdx.x; b < bl * (p - 1); b += blockDim.x) {
                const int t = 1 + b / bl, bb = b - (t - 1) * bl;
                const int line = (int)fdiv((uint32_t)bb, dnb);
                const int loc = bb - line * nb;
                const int j1 = (int)fdiv((uint32_t)loc, drq);
                C *s = src + (size_t)line * n + j1 * rq * p + (loc - j1 * rq);
                if (j1 > 0) s[t * rq] = cx_mul(s[t * rq], tw_get<C, SIGN>(tw, j1 * t * rq));
            }
            __syncthreads();
        }
        // two outputs of two butterflies per thread take four shared-memory
        // reads for four products where one output takes two reads a product
        // (the reads bound the stage: 7 fields 422 x 462, lines 1346 = 2 x 673 and
        // 1386, row pass 464 -> 346 us), where that leaves threads enough busy (73 x
        // 247, lines 567 and 741: 40 us so, 32 one by one)
        if (4 * bl * m >= 3 * (int)blockDim.x)
            generic_sums<C, SIGN, 2>(src, dst, n, bl, L1, p, rq, drq, dnb, tw, a, m);
        else
            generic_sums_1<C, SIGN>(src, dst, n, bl, L1, p, rq, drq, dnb, tw, a, m);
    }
}

// Run all stages with a compile-time transform sign; returns the buffer
// holding the result (a or b).  The caller reads the outputs lo .. lo + cnt - 1
// (mod n; 0 <= lo < n, cnt <= n); others may be left unwritten.
template <typename C, int SIGN>
__device__ C *fft_run_s(C *a, C *b, const FftPlan &pl, int nlines, const C *__restrict__ tw, int lo, int cnt)
{
    int L1 = 1;
    C *src = a, *dst = b;
    for (int q = 0; q < pl.nstages; ++q) {
        const int p = pl.radix[q];
        const int rq = pl.rq[q];
        const FDiv drq = pl.drq[q], dnb = pl.dnb[q];
        __syncthreads();
        switch (p) {
        case 2: stage_p<C, 2, SIGN>(src, dst, pl.n, nlines, L1, rq, drq, dnb, tw); break;
        case 3: stage_p<C, 3, SIGN>(src, dst, pl.n, nlines, L1, rq, drq, dnb, tw); break;
        case 4: stage_p<C, 4, SIGN>(src, dst, pl.n, nlines, L1, rq, drq, dnb, tw); break;
        case 5: stage_p<C, 5, SIGN>(src, dst, pl.n, nlines, L1, rq, drq, dnb, tw); break;
        case 8: stage_p<C, 8, SIGN>(src, dst, pl.n, nlines, L1, rq, drq, dnb, tw); break;
        default: {
            int a = 0, m = p;
            if (q == pl.nstages - 1) {
                a = lo / L1;
                m = min(p, (lo - a * L1 + cnt + L1 - 1) / L1);
            }
            stage_generic<C, SIGN>(src, dst, pl.n, nlines, L1, p, rq, drq, dnb, tw, a, m);
        } break;
        }
        L1 *= p;
        C *t = src;
        src = dst;
        dst = t;
    }
    __syncthreads();
    return src;
}

template <typename C>
__device__ C *fft_run(C *a, C *b, const FftPlan &pl, int nlines, const C *__restrict__ tw, int sign,
                      int lo, int cnt)
{
    return sign > 0 ? fft_run_s<C, 1>(a, b, pl, nlines, tw, lo, cnt)
                    : fft_run_s<C, -1>(a, b, pl, nlines, tw, lo, cnt);
}
