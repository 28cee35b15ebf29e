// Footprint-weighted point measurement (reference: point_measurement,
// src/bldfm/utils.py:80-92, np.sum(f * g)) for a batch of (footprint, flux)
// pairs: out[b] = sum_i f[b][i] g[b][i] in FP64.
//
// HBM (16 bytes read per point, nothing written) and the FP64 pipe bound it about
// evenly: at 2 lanes per clock and SM the pipe passes some 0.53 T instructions/s
// and HBM delivers 0.42 T points/s, 1.25 instructions a point.  A compensated
// sum per point took five (195 us for 64 x 512^2 points, 1.37 TB/s).  Here a
// thread adds 16 points in two chains of 8 FMAs (products unrounded) and only the
// sum of those 16 goes through the compensated accumulator: 1.31 instructions a
// point, 59 us.  Each batch entry is split over the CTAs of one grid row, each
// with a contiguous range; the CTA combines its threads in a fixed order, and the
// cluster or a second kernel (one warp per entry) adds the per-CTA partials in a
// fixed order, so the result is deterministic (no atomics).
//
// Every addition over threads, warps and CTAs keeps its rounding error.  Worst
// case in u = 2^-53 of sum |f g|, at any n: 12 (chain 8, join of the two chains 1,
// compensated sum 2, result 1); a compensated sum per point with a plain tree
// over the threads has 13.  Footprints against flux maps: 64 fields of 512^2
// 5.3e-17, 400 of 300^2 5.2e-17, the rounding of the result itself (5.4e-17 and
// 8.3e-17 with that tree).  numpy's pairwise sum differs at the level of its own
// rounding (about log2(n) eps).
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/bldfm_gb300.h"
#include "tc.cuh"

namespace {

const int MEAS_THREADS = 256;

struct Kahan {
    double s = 0.0, c = 0.0;
    __device__ __forceinline__ void add(double x)
    {
        const double y = __dsub_rn(x, c);
        const double t = __dadd_rn(s, y);
        c = __dsub_rn(__dsub_rn(t, s), y);
        s = t;
    }
};

// A sum that carries its rounding errors along (TwoSum: exact).  An error made in
// one of M equal partial sums weighs 1 / sqrt(M) in the result, so the last
// additions would hold nearly all of it.  The chain from one addition to the
// next is one instruction, Kahan's is four.
struct TwoSum {
    double s = 0.0, e = 0.0;
    __device__ __forceinline__ void add(double x)
    {
        const double t = __dadd_rn(s, x);
        const double b = __dsub_rn(t, s);
        e = __dadd_rn(e, __dadd_rn(__dsub_rn(s, __dsub_rn(t, b)), __dsub_rn(x, b)));
        s = t;
    }
    // lanes l and l + off, for off, off / 2 ... 1, in lane 0
    __device__ __forceinline__ void add_lanes(int off)
    {
        for (; off > 0; off >>= 1) {
            const double s2 = __shfl_down_sync(0xffffffffu, s, off), e2 = __shfl_down_sync(0xffffffffu, e, off);
            add(s2);
            e = __dadd_rn(e, e2);
        }
    }
    __device__ __forceinline__ double sum() const { return __dadd_rn(s, e); }
};

const int MEAS_UNROLL = 8;  // pairs of points per compensated addition
const int MEAS_CTAS = 4;    // resident CTAs per SM the grid is sized for; their 64 registers a thread hold some of
                            // a block's 16 loads of 16 bytes in flight, not all
// Fields of up to 65,536 points take at most eight CTAs, one cluster, which adds
// its partial sums itself: one launch instead of two (31 -> 26 us a call).  With
// more points a CTA than this it takes longer than the second launch (a single
// field of 131,044 points: 46 us with its synchronisation, 43 over the device).
// Batches that leave an entry no more than eight CTAs at any size take it too: 100
// fields of 512^2 132 us (320 with a second launch and a compensated sum per
// point), 305, which get one CTA each, 323 (998), 607 421 (1572), 100 of 1024^2
// 363 (1137).
const int MEAS_CLUSTER = 8, MEAS_CTA_POINTS = 8192;

// not .aligned: thread 0 comes from a branch of its own
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive;\n\tbarrier.cluster.wait;" ::: "memory");
}

// CLUSTER: the grid row is one cluster and writes the entry's sum to part[b],
// else every CTA its partial sum.
template <bool CLUSTER>
__global__ void __launch_bounds__(MEAS_THREADS, MEAS_CTAS)
    meas_partial_kernel(const double *__restrict__ f, const double *__restrict__ g, int64_t n, int64_t stride,
                        double *__restrict__ part)
{
    const int b = blockIdx.y;
    const double *fb = f + (size_t)b * stride, *gb = g + (size_t)b * stride;
    Kahan k;
    const bool vec = ((((uintptr_t)fb) ^ ((uintptr_t)gb)) & 15) == 0;
    if (vec) {
        // both at the same 8-byte phase: one leading point at most, then pairs
        const int lead = (((uintptr_t)fb) & 15) != 0 && n > 0 ? 1 : 0;
        const int64_t n2 = (n - lead) / 2;
        const double2 *f2 = (const double2 *)(fb + lead), *g2 = (const double2 *)(gb + lead);
        // this CTA's pairs
        const int64_t per = (n2 + gridDim.x - 1) / gridDim.x;
        const int64_t lo = (int64_t)blockIdx.x * per, hi = min(n2, lo + per);
        int64_t i = lo + threadIdx.x;
        for (; i + (MEAS_UNROLL - 1) * MEAS_THREADS < hi; i += MEAS_UNROLL * MEAS_THREADS) {
            double2 a[MEAS_UNROLL], c[MEAS_UNROLL];
#pragma unroll
            for (int u = 0; u < MEAS_UNROLL; ++u) {
                a[u] = __ldcs(f2 + i + u * MEAS_THREADS);
                c[u] = __ldcs(g2 + i + u * MEAS_THREADS);
            }
            double s0 = a[0].x * c[0].x, s1 = a[0].y * c[0].y;
#pragma unroll
            for (int u = 1; u < MEAS_UNROLL; ++u) {
                s0 = fma(a[u].x, c[u].x, s0);
                s1 = fma(a[u].y, c[u].y, s1);
            }
            k.add(__dadd_rn(s0, s1));
        }
        for (; i < hi; i += MEAS_THREADS) {
            const double2 a = __ldcs(f2 + i), c = __ldcs(g2 + i);
            k.add(fma(a.x, c.x, __dmul_rn(a.y, c.y)));
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            if (lead) k.add(__dmul_rn(fb[0], gb[0]));
            if ((n - lead) & 1) k.add(__dmul_rn(fb[n - 1], gb[n - 1]));
        }
    } else {
        const int64_t step = (int64_t)gridDim.x * MEAS_THREADS;
        for (int64_t i = (int64_t)blockIdx.x * MEAS_THREADS + threadIdx.x; i < n; i += step)
            k.add(__dmul_rn(__ldg(fb + i), __ldg(gb + i)));
    }
    // the threads' sums with their errors: eight per lane of one warp, then its lanes
    __shared__ double ss[MEAS_THREADS];
    ss[threadIdx.x] = __dadd_rn(k.s, -k.c);
    __syncthreads();
    if (threadIdx.x < 32) {
        TwoSum t;
        t.s = ss[threadIdx.x];
#pragma unroll
        for (int w = 1; w < MEAS_THREADS / 32; ++w) t.add(ss[threadIdx.x + 32 * w]);
        t.add_lanes(16);
        if (threadIdx.x == 0) ss[0] = t.sum();
    }
    if (CLUSTER) {
        cluster_sync();
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            TwoSum t;
            for (unsigned r = 0; r < gridDim.x; ++r) {
                uint32_t a;
                double x;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(tc_smem(ss)), "r"(r));
                asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x) : "r"(a) : "memory");
                t.add(x);
            }
            part[b] = t.sum();
        }
        cluster_sync();  // no CTA leaves while its sum may still be read
    } else if (threadIdx.x == 0) {
        part[(size_t)b * gridDim.x + blockIdx.x] = ss[0];
    }
}

// CTAs per entry: enough points for each, and one wave over the device
int meas_ctas(int64_t n, int32_t nbatch)
{
    int dev = 0, nsm = 152;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    int64_t per = (n + MEAS_THREADS * 4 - 1) / (MEAS_THREADS * 4);
    const int64_t want = (int64_t)nsm * MEAS_CTAS / nbatch;
    if (per > want) per = want;
    if (n <= (int64_t)MEAS_CLUSTER * MEAS_CTA_POINTS && per > MEAS_CLUSTER) per = MEAS_CLUSTER;
    if (per < 1) per = 1;
    if (per > 65535) per = 65535;
    return (int)per;
}

// One warp per batch entry: lane l adds the partials l, l + 32, ... (one
// thread's chain over all 600 partials of a single field took longer than the
// field's own pass), then the lanes in a fixed tree order.
__global__ void __launch_bounds__(128) meas_final_kernel(const double *__restrict__ part, int nparts, int nbatch,
                                                         double *__restrict__ out)
{
    const int b = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (b >= nbatch) return;
    TwoSum k;
    for (int i = lane; i < nparts; i += 32) k.add(part[(size_t)b * nparts + i]);
    k.add_lanes(nparts > 16 ? 16 : nparts > 8 ? 8 : 4);  // as many levels as lanes hold partials
    if (lane == 0) out[b] = k.sum();
}

// One CTA waits on an mbarrier that nothing arrives at, with an iteration
// limit: the bounded-wait path every waiting kernel takes on a timeout.  The
// elapsed global-timer nanoseconds of the wait go to ns[0].
__global__ void wait_timeout_kernel(long limit, int *status, long long *ns)
{
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        tc_mbar_init(&bar, 1);
        tc_fence_init();
    }
    __syncthreads();
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    const uint32_t a = tc_smem(&bar);
    uint32_t done = 0;
    for (long it = 0; it < limit && !done; ++it) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(0u)
            : "memory");
    }
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
    if (__syncthreads_or(!done) && threadIdx.x == 0) {
        *status = BLDFM_ERR_TIMEOUT;
        *ns = (long long)(t1 - t0);
    }
}

}  // namespace

extern "C" {

// Self-check of the failure-detection path (no reference counterpart): a
// kernel whose wait can never complete gives up after `limit` polls and
// reports BLDFM_ERR_TIMEOUT in *status_host, with the time the wait took in
// *wait_ns_host; the context stays usable.
int bldfm_selftest_wait_timeout(int64_t limit, int32_t *status_host, int64_t *wait_ns_host)
{
    if (!status_host || !wait_ns_host || limit < 1 || limit > ((int64_t)1 << 20)) return BLDFM_ERR_ARG;
    void *d = nullptr;
    if (cudaMalloc(&d, 16) != cudaSuccess) return BLDFM_ERR_CUDA;
    int rc = BLDFM_OK;
    if (cudaMemset(d, 0, 16) != cudaSuccess) rc = BLDFM_ERR_CUDA;
    if (rc == BLDFM_OK) {
        wait_timeout_kernel<<<1, 64>>>((long)limit, (int *)d, (long long *)((char *)d + 8));
        if (cudaDeviceSynchronize() != cudaSuccess) rc = BLDFM_ERR_CUDA;
    }
    long long h[2] = {0, 0};
    if (rc == BLDFM_OK && cudaMemcpy(h, d, 16, cudaMemcpyDeviceToHost) != cudaSuccess) rc = BLDFM_ERR_CUDA;
    *status_host = (int32_t)(int)h[0];
    *wait_ns_host = (int64_t)h[1];
    cudaFree(d);
    return rc;
}

// Scratch bytes bldfm_point_measurement needs for nbatch entries of n points.
int64_t bldfm_point_measurement_workspace(int64_t n, int32_t nbatch)
{
    if (n < 0 || nbatch < 1) return -1;
    return (int64_t)meas_ctas(n, nbatch) * nbatch * (int64_t)sizeof(double);
}

int bldfm_point_measurement(const double *f_dev, const double *g_dev, int64_t n, int64_t stride, int32_t nbatch,
                            double *out_dev, void *workspace_dev, size_t workspace_bytes, void *stream)
{
    if (!f_dev || !g_dev || !out_dev || n < 0 || stride < n || nbatch < 1 || nbatch > 65535) return BLDFM_ERR_ARG;
    const int64_t need = bldfm_point_measurement_workspace(n, nbatch);
    if (!workspace_dev || need < 0 || (int64_t)workspace_bytes < need) return BLDFM_ERR_WORKSPACE;
    if (((uintptr_t)workspace_dev & 7) != 0) return BLDFM_ERR_ARG;
    const int per = meas_ctas(n, nbatch);
    cudaStream_t st = (cudaStream_t)stream;
    double *part = (double *)workspace_dev;
    if (per <= MEAS_CLUSTER) {
        cudaLaunchAttribute at = {};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = per;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(per, nbatch);
        cfg.blockDim = dim3(MEAS_THREADS);
        cfg.stream = st;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        // a refused launch also leaves its error behind, which the return takes
        (void)cudaLaunchKernelEx(&cfg, meas_partial_kernel<true>, f_dev, g_dev, n, stride, out_dev);
    } else {
        meas_partial_kernel<false><<<dim3(per, nbatch), MEAS_THREADS, 0, st>>>(f_dev, g_dev, n, stride, part);
        meas_final_kernel<<<(nbatch + 3) / 4, 128, 0, st>>>(part, per, nbatch, out_dev);
    }
    return cudaGetLastError() == cudaSuccess ? BLDFM_OK : BLDFM_ERR_CUDA;
}

}  // extern "C"
