// kernels.cu -- sm_103a kernels of the GB300 PairHMM.
//
// The recurrence is LoglessPairHMM's (src/main/java/org/broadinstitute/hellbender/utils/pairhmm/
// LoglessPairHMM.java:47-67): for matrix row i (read position i-1) and column j (haplotype position j-1),
//   M(i,j) = prior(i,j) * (M(i-1,j-1)*MM_i + I(i-1,j-1)*IM_i + D(i-1,j-1)*IM_i)
//   I(i,j) = M(i-1,j)*MI_i + I(i-1,j)*II_i
//   D(i,j) = M(i,j-1)*MD_i + D(i,j-1)*DD_i
// with D(0,j) = scale/H, every other row-0 and column-0 entry 0, and
// log10 L = log10(sum_j M(R,j) + I(R,j)) - log10(scale).
//
// Three kernels:
//  * fp32_bucket_kernel<K, MULTI> (fp32_bucket.cuh; here and in fp32_mixed.cu): the batched FP32 forward.  One warp runs a read-pair task: two reads of
//    one region, packed into the .x/.y halves of float2 so every cell update is a packed FFMA2/FMUL2/FADD2,
//    against all (or a chunk of) the region's haplotypes streamed back to back.  Lane l owns K consecutive
//    rows; at step s it computes column c = s - 2l, receiving the row above from lane l-1 by __shfl_up_sync
//    (an anti-diagonal wavefront with a skew of two columns per lane, so that a value shuffled at the start of
//    a step is consumed one step later and the shuffle's latency stays off the per-step chain); lane l-1 hands
//    lane l two packed values per step, its row 0's I~ at a column and the inner sum b I~ + c D~ + M~ of its
//    row 0's M~ at the next column, computed with lane l's row-0 coefficients, instead of three raw states
//    (K >= 2).  Each read is followed by two accumulator rows that sum the last row over
//    the haplotype (row_coef), and padded at the top with "dummy" rows that reproduce the row-0 boundary, so
//    the accumulator rows always sit in lane 31's last two slots.  Reads longer than 32*K rows run
//    as several strips whose boundary row goes through per-warp global scratch (and a ring in shared memory).  Each row's states are
//    rescaled so a cell costs 5 FMA-pipe operations instead of 8: with a_0 = 1, a_i = a_{i-1} / MM_i,
//       M~ = a_i M,   I~ = (a_{i-1} / MI_i) I,   D~ = (a_i / MD_i) D,
//    the recurrence becomes
//       M~ = prior * fma(I~_diag, b_i, fma(D~_diag, c_i, M~_diag))
//       I~ = fma(I~_up, e_i, M~_up)
//       D~ = fma(D~_left, DD_i, M~_left)
//    with b_i = IM_i MI_{i-1} / (MM_i MM_{i-1}), c_i = IM_i MD_{i-1} / MM_i, e_i = II_i MI_{i-1} / (MI_i MM_{i-1})
//    (MM_0 = MI_0 = MD_0 = 1) and  M_R + I_R = (M~_R + I~_R MI_R / MM_R) / a_R.  Only ratios of adjacent rows'
//    coefficients appear; log2 a_R is summed per read once per upload (read_scale_kernel, in FP64 and in an order
//    fixed by the read, so a read's result is the same whatever task or batch it runs in).  Reads whose I~ could
//    outgrow FP32 (steeply rising insertion penalties) or whose MM is 0 are sent to FP64 by the host.
//    Scale 2^120; a sum below GHMM_FP32_RERUN_THRESHOLD (or not finite) queues the pair for FP64.
//  * fp64_queue_kernel<RESCALED> (fp64.cu): the FP64 wavefront, used for reruns and double-precision mode: a rescaled
//    tier (5 DP operations per cell) and an exact unscaled tier (scale 2^1020, LoglessPairHMM's magnitudes) for results
//    near the bottom of the FP64 range.
//  * plain_fp64_kernel: the plain form, one pair per thread block sweeping anti-diagonals through shared
//    memory with a block barrier per diagonal, Java's operation order, one launch per region.
#include <cuda_runtime.h>

#include <cstdint>

namespace {
constexpr bool kMixedTasks = false;
}
#include "fp32_bucket.cuh"

namespace ghmm {

// Per read: log2 a_R = sum over its positions of -log2 MM (the FP32 pass's row rescaling, with the float
// matchToMatch values its coefficients use, from a host-built FP64 table), summed in FP64 in an order fixed by the
// read alone, so that a read's
// result does not depend on the task, rows per lane or batch it runs in.  Stored as (2^-(la - n), n), n = round(la).
// One warp per read; computed once per upload (after the read preparation for raw batches).
__global__ void read_scale_kernel(DevTables T, DevBatch B, int64_t n_reads, float2 *scale) {
    const int lane = threadIdx.x & 31;
    for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n_reads;
         r += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t off = B.read_off[r], len = B.read_off[r + 1] - off;
        double la = 0.0;
        for (int64_t p = lane; p < len; p += 32)
            la += __ldg(T.lm2m_d + B.ins[off + p] * 128 + B.dels[off + p]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) la += __shfl_xor_sync(kFull, la, o);
        if (lane == 0) {
            const double n = rint(la);
            scale[r] = make_float2((float)exp2(n - la), (float)n);
        }
    }
}

// Final log10 un-scaling of the FP32 pass, in FP64: out = log10(t) - log10(a_R) - log10(2^120).  Runs before the FP64
// queue kernel, which then overwrites the pairs it recomputes (their slots hold no accepted sum).
__global__ void finalize_fp32_kernel(double *out, const int64_t *n_out) {
    const int64_t n = *n_out;
    const double log10_2 = 0.30102999566398120;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float2 v = reinterpret_cast<const float2 *>(out)[i];  // (t, log2 a_R), see emit_fp32
        out[i] = log10((double)v.x) - (double)v.y * log10_2 - kLog10Scale32;
    }
}

// ---------------------------------------------------------------------------------------------------
// Plain FP64 form: one (read, haplotype) pair per 256-thread block; thread t owns rows t+1+256m (m<ROWS:
// 4 rows for reads up to 1024 bases, 8 up to 2048); three rolling anti-diagonals of M, I, D in shared
// memory; one barrier per diagonal; Java's order of operations (no fused multiply-add), so the sums equal
// the FP64 oracle's.
constexpr int kPlainThreads = 256;

template <int kPlainRows>
__global__ void __launch_bounds__(kPlainThreads) plain_fp64_kernel(DevTables T, DevBatch B, int region, int nh) {
    extern __shared__ double sm[];
    const int pair = blockIdx.x;
    const int64_t read = B.region_read_off[region] + pair / nh;
    const int64_t hap = B.region_hap_off[region] + pair % nh;
    const int64_t roff = B.read_off[read];
    const int R = (int)(B.read_off[read + 1] - roff);
    const int64_t hoff = B.hap_off[hap];
    const int H = (int)(B.hap_off[hap + 1] - hoff);
    const int64_t out_index = B.out_off[region] + pair;
    if (R == 0 || H == 0) {
        if (threadIdx.x == 0) B.out[out_index] = -INFINITY;
        return;
    }
    const int W = R + 1;
    double *Mb = sm, *Ib = sm + 3 * W, *Db = sm + 6 * W;  // [3][W] each
    const double init = B.hap_init_d[hap];
    double t_mm[kPlainRows], t_im[kPlainRows], t_mi[kPlainRows], t_ii[kPlainRows], t_md[kPlainRows];
    double p_m[kPlainRows], p_e[kPlainRows];
    uint8_t xb[kPlainRows];
#pragma unroll
    for (int m = 0; m < kPlainRows; ++m) {
        const int i = threadIdx.x + 1 + m * kPlainThreads;
        if (i <= R) {
            const int p = i - 1;
            const uint8_t q = B.quals[roff + p], ins = B.ins[roff + p], del = B.dels[roff + p];
            const uint8_t gcp = B.gcp[roff + p];
            t_mm[m] = T.m2m_d[ins * 128 + del];
            t_im[m] = T.prob_d[gcp];
            t_mi[m] = T.err_d[ins];
            t_ii[m] = T.err_d[gcp];
            t_md[m] = T.err_d[del];
            p_m[m] = T.prob_d[q];
            p_e[m] = T.err3_d[q];
            xb[m] = B.bases[roff + p];
        } else {
            t_mm[m] = t_im[m] = t_mi[m] = t_ii[m] = t_md[m] = p_m[m] = p_e[m] = 0.0;
            xb[m] = 0;
        }
    }
    for (int b = 0; b < 3; ++b)
        for (int i = threadIdx.x; i < W; i += kPlainThreads) {
            Mb[b * W + i] = 0.0;
            Ib[b * W + i] = 0.0;
            Db[b * W + i] = (i == 0) ? init : 0.0;
        }
    __syncthreads();
    double sum = 0.0;
    for (int d = 2; d <= R + H; ++d) {
        const int cur = d % 3, p1 = (d + 2) % 3, p2 = (d + 1) % 3;
#pragma unroll
        for (int m = 0; m < kPlainRows; ++m) {
            const int i = threadIdx.x + 1 + m * kPlainThreads;
            if (i > R) continue;
            const int j = d - i;
            if (j == 0) {  // column-0 boundary
                Mb[cur * W + i] = 0.0;
                Ib[cur * W + i] = 0.0;
                Db[cur * W + i] = 0.0;
                continue;
            }
            if (j < 1 || j > H) continue;
            const uint8_t y = B.hap_bases[hoff + j - 1];
            const double prior = (xb[m] == y || xb[m] == 'N' || y == 'N') ? p_m[m] : p_e[m];
            const double mdiag = Mb[p2 * W + i - 1], idiag = Ib[p2 * W + i - 1], ddiag = Db[p2 * W + i - 1];
            const double mup = Mb[p1 * W + i - 1], iup = Ib[p1 * W + i - 1];
            const double mleft = Mb[p1 * W + i], dleft = Db[p1 * W + i];
            const double mv = __dmul_rn(prior, __dadd_rn(__dadd_rn(__dmul_rn(mdiag, t_mm[m]), __dmul_rn(idiag, t_im[m])),
                                                         __dmul_rn(ddiag, t_im[m])));
            const double iv = __dadd_rn(__dmul_rn(mup, t_mi[m]), __dmul_rn(iup, t_ii[m]));
            const double dv = __dadd_rn(__dmul_rn(mleft, t_md[m]), __dmul_rn(dleft, t_ii[m]));
            Mb[cur * W + i] = mv;
            Ib[cur * W + i] = iv;
            Db[cur * W + i] = dv;
            if (i == R) sum = __dadd_rn(sum, __dadd_rn(mv, iv));
        }
        __syncthreads();
    }
    if ((int)threadIdx.x == (R - 1) % kPlainThreads) B.out[out_index] = log10(sum) - kLog10Scale64;
}

// ---------------------------------------------------------------------------------------------------
// FP32 / FP64 pipe peak probes: register-resident chains, 8 independent per thread.
template <int N>
__global__ void peak_ffma_kernel(float *out, int iters, float x, float y) {
    float a[N];
#pragma unroll
    for (int i = 0; i < N; ++i) a[i] = threadIdx.x * 1e-7f + i;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int i = 0; i < N; ++i) a[i] = fmaf(a[i], x, y);
    }
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) s += a[i];
    if (s == 12345.678f) out[threadIdx.x] = s;
}

template <int N>
__global__ void peak_ffma2_kernel(float *out, int iters, float x, float y) {
    float2 a[N];
#pragma unroll
    for (int i = 0; i < N; ++i) a[i] = make_float2(threadIdx.x * 1e-7f + i, threadIdx.x * 2e-7f + i);
    const float2 xx = make_float2(x, x), yy = make_float2(y, y);
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int i = 0; i < N; ++i) a[i] = __ffma2_rn(a[i], xx, yy);
    }
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) s += a[i].x + a[i].y;
    if (s == 12345.678f) out[threadIdx.x] = s;
}

template <int N>
__global__ void peak_dfma_kernel(double *out, int iters, double x, double y) {
    double a[N];
#pragma unroll
    for (int i = 0; i < N; ++i) a[i] = threadIdx.x * 1e-7 + i;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int i = 0; i < N; ++i) a[i] = fma(a[i], x, y);
    }
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) s += a[i];
    if (s == 12345.678) out[threadIdx.x] = s;
}

// ---------------------------------------------------------------------------------------------------
int launch_fp32_bucket(const DevTables &t, const DevBatch &b, int key, int grid, int block, cudaStream_t s) {
    return bucket_mixed(key) ? launch_fp32_mixed(t, b, key, grid, block, s) : launch_fp32_form(t, b, key, grid, block, s);
}

int fp32_kernel_occupancy(int key, int block, int *blocks_per_sm) {
    return bucket_mixed(key) ? fp32_mixed_occupancy(key, block, blocks_per_sm) : fp32_form_occupancy(key, block, blocks_per_sm);
}

int launch_read_scale(const DevTables &t, const DevBatch &b, int64_t n_reads, float2 *scale, int sm_count,
                      cudaStream_t s) {
    if (n_reads <= 0) return 0;
    const int64_t want = (n_reads + 7) / 8;  // 8 warps per 256-thread block
    read_scale_kernel<<<(int)(want < (int64_t)sm_count * 8 ? want : (int64_t)sm_count * 8), 256, 0, s>>>(t, b, n_reads,
                                                                                                          scale);
    return (int)cudaGetLastError();
}

int launch_finalize_fp32(double *out, const int64_t *n_out, int sm_count, cudaStream_t s) {
    finalize_fp32_kernel<<<sm_count * 4, 256, 0, s>>>(out, n_out);
    return (int)cudaGetLastError();
}

// Shared memory: three diagonals of M, I, D over R+1 rows, sized by the region's longest read.
int launch_plain_region(const DevTables &t, const DevBatch &b, int region, int n_reads, int n_haps,
                              int max_read_len, cudaStream_t s) {
    if (n_reads <= 0 || n_haps <= 0) return 0;
    if (max_read_len > kPlainMaxRead) return (int)cudaErrorInvalidValue;
    const size_t smem = sizeof(double) * 9 * (size_t)(max_read_len + 1);
    const bool wide = max_read_len > 4 * kPlainThreads;
    if (smem > 48 * 1024) {
        cudaError_t e = wide ? cudaFuncSetAttribute(plain_fp64_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
                             : cudaFuncSetAttribute(plain_fp64_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    if (wide)
        plain_fp64_kernel<8><<<n_reads * n_haps, kPlainThreads, smem, s>>>(t, b, region, n_haps);
    else
        plain_fp64_kernel<4><<<n_reads * n_haps, kPlainThreads, smem, s>>>(t, b, region, n_haps);
    return (int)cudaGetLastError();
}

int measure_peaks_device(int sm_count, double *fp32, double *fp32x2, double *fp64, cudaStream_t s) {
    float *fo = nullptr;
    double *dout = nullptr;
    if (cudaMalloc(&fo, 1024 * sizeof(float)) != cudaSuccess) return (int)cudaErrorMemoryAllocation;
    if (cudaMalloc(&dout, 1024 * sizeof(double)) != cudaSuccess) {
        cudaFree(fo);
        return (int)cudaErrorMemoryAllocation;
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int block = 256, grid = sm_count * 8;
    constexpr int N = 8;
    const double threads = (double)grid * block;
    float ms = 0.f;
    int err = 0;
    // best of three timed launches after a warm-up, so a clock still ramping up does not lower the peak
    auto timeit = [&](auto launch, int iters, double flops_per_iter_thread, double *res) {
        launch(iters / 8);
        double best = 0.0;
        for (int rep = 0; rep < 3; ++rep) {
            cudaEventRecord(e0, s);
            launch(iters);
            cudaEventRecord(e1, s);
            cudaEventSynchronize(e1);
            cudaEventElapsedTime(&ms, e0, e1);
            const double v = threads * iters * flops_per_iter_thread / (ms * 1e-3) / 1e12;
            if (v > best) best = v;
        }
        if (res) *res = best;
        if (cudaGetLastError() != cudaSuccess) err = 1;
    };
    timeit([&](int it) { peak_ffma_kernel<N><<<grid, block, 0, s>>>(fo, it, 0.999999f, 1e-6f); }, 1 << 16,
           2.0 * N, fp32);
    timeit([&](int it) { peak_ffma2_kernel<N><<<grid, block, 0, s>>>(fo, it, 0.999999f, 1e-6f); }, 1 << 15,
           4.0 * N, fp32x2);
    timeit([&](int it) { peak_dfma_kernel<N><<<grid, block, 0, s>>>(dout, it, 0.999999, 1e-6); }, 1 << 11,
           2.0 * N, fp64);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(fo);
    cudaFree(dout);
    return err ? (int)cudaErrorLaunchFailure : 0;
}

}  // namespace ghmm
