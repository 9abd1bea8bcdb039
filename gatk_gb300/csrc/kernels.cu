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
//  * fp32_bucket_kernel<K, MULTI>: the batched FP32 forward.  One warp runs a read-pair task: two reads of
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
#include <cfloat>
#include <cstdint>
#include <type_traits>

#include "../../include/ghmm.h"
#include "fp32_rows.cuh"
#include "ghmm_internal.h"

namespace ghmm {

namespace {

constexpr int kPlain = 0, kReset = 1, kZero = 2, kCheck = 3;  // kinds of wavefront steps of the FP32 kernel

// t = a_R (M_R + I_R) summed over the haplotype (scaled by 2^120); the read's scale (s, n) from read_scale_kernel
// splits log2 a_R = n - log2 s into an integer n and a factor s in [2^-1/2, 2^1/2].  Accepted sums are stored raw
// as the float pair (t s, n) in the output slot; finalize_fp32_kernel turns them into log10 in FP64 with every lane
// busy, rather than one lane per warp running the FP64 log10 here on the 1/64-rate FP64 pipe.
__device__ __forceinline__ void emit_fp32(const DevBatch &B, float t, float2 scale, int read, int hap,
                                          int64_t out_index) {
    t *= scale.x;
    const float la = scale.y;
    const bool forced = B.force_rerun_every > 0 && out_index % B.force_rerun_every == 0;  // test hook
    if (t > 0.f && t <= FLT_MAX && log2f(t) - la >= kLog2Threshold && !forced) {
        reinterpret_cast<float2 *>(B.out)[out_index] = make_float2(t, la);
    } else {
        const int idx = atomicAdd(&B.counters[1], 1);
        if ((int64_t)idx < B.rerun_capacity) {
            B.rerun[idx].read = read;
            B.rerun[idx].hap = hap;
        } else {
            atomicExch(&B.counters[3], 1);
        }
    }
}

}  // namespace

// Blocks of 128 threads the FP32 kernel asks ptxas to fit per SM (register budget 65536 / (128 * n)).  K <= 5 fits
// four without spilling (126 registers at K = 5: 0.4 % faster than three); K = 6 and 7 at four spill a little and
// ran 1-2 % slower, K = 8 spills 600 bytes.
template <int K>
struct Fp32MinBlocks {
    static constexpr int value = K >= 6 ? 3 : 4;
};

// The bucket's task range and cursor live in device memory (B.bucket_info, B.counters), so the launch
// arguments do not depend on the batch and a captured CUDA graph can be replayed for every batch.
// MIXED: tasks of short and long haplotypes (kBucketMixed).  A kernel of its own, since the loops of a third form in one
// kernel make the compiler's code for the other two up to 4 % slower.
template <int K, bool MULTI, bool MIXED>
__global__ void __launch_bounds__(128, Fp32MinBlocks<K>::value) fp32_bucket_kernel(DevTables T, DevBatch B) {
    constexpr int KEY = K + (MIXED ? kBucketMixed : 0) + (MULTI ? kBucketMulti : 0);
    const int task_begin = B.bucket_info[KEY], task_count = B.bucket_info[kNumBucketKeys + KEY];
    const int counter_slot = kCounterBucketBase + KEY;
    constexpr int S = 32 * K;
    const int lane = threadIdx.x & 31;
    // Per-warp prior table in shared memory: prior[k/2][base][lane] holds rows k and k+1 as (read A, read B,
    // read A, read B), base index A,C,G,T,N = 0..4.  One 128-bit load per row pair and step replaces four
    // compares and four selects.
    constexpr int KP = (K + 1) / 2;  // row pairs
    extern __shared__ float4 prior_smem4[];
    float4 *prior_tbl4 = prior_smem4 + (size_t)(threadIdx.x >> 5) * (KP * kBases * 32) + lane;
    float2 *prior_tbl2 = reinterpret_cast<float2 *>(prior_tbl4);
    const int64_t warp_global = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    // Strip boundary (MULTI): per column lane 31's hand-over (I~, M~ inner sum) as one float4 in global scratch.  Lane 0 of
    // the next strip reads it from a ring of 64 columns in shared memory that the warp fills 32 columns at a time, loaded
    // 32 steps before that; read from global memory column by column, a step ahead, the load's latency was in every step
    // (FP32 pass of reads of 510 bases x haplotypes of 600: 3,110 GCUPS, with the ring 3,845).
    float4 *scratch = nullptr, *ring = nullptr;
    if (MULTI) {
        scratch = B.scratch32 + warp_global * B.scratch32_cols;
        ring = prior_smem4 + 4 * (KP * kBases * 32) + (threadIdx.x >> 5) * 64;
    }

    for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(&B.counters[counter_slot], 1);
        t = __shfl_sync(kFull, t, 0);
        if (t >= task_count) break;
        const F32Task task = B.tasks[task_begin + t];
        const int ra = task.read_a, rb = task.read_b;
        const int64_t off_a = B.read_off[ra];
        const int len_a = (int)(B.read_off[ra + 1] - off_a);
        int64_t off_b = 0;
        int len_b = 0;
        if (rb >= 0) {
            off_b = B.read_off[rb];
            len_b = (int)(B.read_off[rb + 1] - off_b);
        }
        const int region = task.region;
        const int64_t hap0 = B.region_hap_off[region];
        const int nh = (int)(B.region_hap_off[region + 1] - hap0);
        const int64_t rr0 = B.region_read_off[region];
        const int64_t out_a = B.out_off[region] + (int64_t)(ra - rr0) * nh - hap0;
        const int64_t out_b = B.out_off[region] + (int64_t)(rb - rr0) * nh - hap0;
        const int64_t col0 = B.hap_off[task.hap_begin];
        const int ncols = (int)(B.hap_off[task.hap_end] - col0);
        const uint8_t *stream = B.hap_code + col0;
        const int nstrips = MULTI ? task.nstrips : 1;
        bool long_haps = true;
        if constexpr (!MIXED) {
            for (int h = task.hap_begin + lane; h < task.hap_end; h += 32)
                long_haps &= B.hap_off[h + 1] - B.hap_off[h] >= kShortHapCols;
            long_haps = __all_sync(kFull, long_haps);
        }

        for (int strip = 0; strip < nstrips; ++strip) {
            float2 cb[K], cc[K], ce[K], cdd[K];
            __syncwarp();  // the previous strip's steps have finished reading this warp's table
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int slot = strip * S + lane * K + k;
                const RowCoef a = row_coef(T, B, off_a, len_a, slot - task.pad_a);
                const RowCoef b = row_coef(T, B, off_b, rb >= 0 ? len_b : 0, slot - task.pad_b);
                cb[k] = make_float2(a.b, b.b);
                cc[k] = make_float2(a.c, b.c);
                ce[k] = make_float2(a.e, b.e);
                cdd[k] = make_float2(a.dd, b.dd);
#pragma unroll
                for (int h = 0; h < kBases; ++h) {
                    const uint32_t hm = kBaseMask[h];
                    prior_tbl2[((k / 2) * kBases + h) * 64 + (k & 1)] =
                        make_float2((a.code & hm) ? a.pm : a.pe, (b.code & hm) ? b.pm : b.pe);
                }
            }
            // row-0 coefficients of the lane below (lane 31: of the next strip's first row), with which this lane
            // hands it its row 0's I~ and M~ inner sum instead of three raw states
            float2 b0n = shfl_down2(cb[0]), c0n = shfl_down2(cc[0]), e0n = shfl_down2(ce[0]);
            if (lane == 31) {
                b0n = c0n = e0n = zero2();
                if (MULTI && strip + 1 < nstrips) {
                    const int slot = (strip + 1) * S;
                    const RowCoef a = row_coef(T, B, off_a, len_a, slot - task.pad_a);
                    const RowCoef b = row_coef(T, B, off_b, rb >= 0 ? len_b : 0, slot - task.pad_b);
                    b0n = make_float2(a.b, b.b);
                    c0n = make_float2(a.c, b.c);
                    e0n = make_float2(a.e, b.e);
                }
            }
            __syncwarp();
            float2 Mp[K], Ip[K], Dp[K];
#pragma unroll
            for (int k = 0; k < K; ++k) Mp[k] = Ip[k] = Dp[k] = zero2();
            float2 gW = zero2();   // row 0's M~ inner sum consumed this step (the diagonal input of row 0)
            float2 w0 = zero2();   // lane 0, strip 0: the row-0 boundary's inner sum c_0 X
            // Lane l runs column s - 2l at step s (a skew of two columns per lane), so what lane l-1 hands over
            // at the end of a step is shuffled at the start of the next one and consumed a step later: the
            // shuffle's latency is off the per-step chain (the I~ recurrence down the lane's rows).
            float2 pendV = zero2();                     // I~ of row 0 for next step's column
            float2 pendW1 = zero2(), pendW2 = zero2();  // row 0's M~ inner sums for the next two steps
            int hap = task.hap_begin - 1;
            const bool last_strip = (strip == nstrips - 1);
            float4 block = make_float4(0.f, 0.f, 0.f, 0.f);  // later strips: the lane's column of the ring's next 32
            auto boundary = [&](int c) {
                return MULTI && strip > 0 && c < ncols ? scratch[c] : make_float4(0.f, 0.f, 0.f, 0.f);
            };
            float2 nxV = zero2(), nxW = zero2(), l0W = zero2();  // later strips, lane 0: the next step's entry, the last W
            if (MULTI && strip > 0) {
                const float4 v = boundary(lane);
                ring[lane] = v;
                block = boundary(32 + lane);
                nxV = make_float2(v.x, v.y);  // (lane 0's: column 0)
                nxW = make_float2(v.z, v.w);
            }
            float2 sV = zero2(), sW = zero2();  // what this lane hands the lane below at the end of a step
            const int nsteps = ncols + 62;
            // column code of the next step, loaded one step ahead (the code plane has kCodePad bytes on
            // both sides, so columns just outside the stream are readable; CHK steps mask them)
            uint32_t code_next = (uint32_t)__ldg(stream - 2 * lane);
            // before the step s = 0 mod 32 of a later strip: columns s + 32 .. s + 63 into the half of the ring that columns
            // s - 32 .. s - 1 had
            auto refill = [&](const int s) {
                if (!MULTI || strip == 0 || (s & 31) != 0) return;
                __syncwarp();
                ring[(s + 32 + lane) & 63] = block;
                __syncwarp();
                block = boundary(s + 64 + lane);
            };
            // lane 31 at a haplotype's last column (K >= 2): the sums of both reads
            auto emit = [&](const int hap) {
                const float2 t = add2(add2(Dp[K - 1], Mp[K - 1]), Ip[K >= 2 ? K - 2 : 0]);
                emit_fp32(B, t.x, __ldg(B.read_scale + ra), ra, hap, out_a + hap);
                if (rb >= 0) emit_fp32(B, t.y, __ldg(B.read_scale + rb), rb, hap, out_b + hap);
            };
            // One wavefront step.  kPlain: no lane starts or ends a haplotype.  kReset: lane `first` is at the first column
            // of a haplotype with row-0 value h_init; kZero: the same for a lane below all dummy rows.  kCheck: any lane may be outside the stream (not started, or
            // finished), at a first column, or at a last one (lane 31 emits), as the column codes say.
            auto step = [&](const int s, auto mode_tag, const int first, const float h_init) {
                constexpr int MODE = decltype(mode_tag)::value;
                constexpr bool CHK = MODE == kCheck;
                const int c = s - 2 * lane;
                bool valid = true;
                uint32_t code = code_next;
                code_next = (uint32_t)__ldg(stream + c + 1);
                if constexpr (CHK) {
                    valid = (c >= 0) && (c < ncols);
                    code = valid ? code : 0u;
                }
                // Lane l-1's hand-over from its last step (its column c + 1): shuffled now, consumed next step
                // (I~) and the step after (the inner sum for column c + 2).  Shuffled before this lane resets its
                // own state at a haplotype start, since lane l+1 still needs this lane's previous column.
                const float2 shV = shfl_up2(sV);
                const float2 shW = shfl_up2(sW);
                float2 uV = pendV;  // I~ of this lane's row 0 at this column
                gW = pendW2;        // row 0's M~ inner sum for this column
                pendV = shV;
                pendW2 = pendW1;
                pendW1 = shW;
                // lane 0 takes the row-0 boundary (strip 0) or the previous strip's last row instead
                // (selects on the ALU pipe, not multiplies on the FMA pipe)
                if (MULTI && strip > 0) {
                    if (lane == 0) {
                        uV = nxV;
                        gW = l0W;
                        l0W = nxW;
                    }
                    const float4 v = ring[(s + 1) & 63];
                    nxV = make_float2(v.x, v.y);
                    nxW = make_float2(v.z, v.w);
                } else if (lane == 0) {
                    uV = zero2();
                }
                if constexpr (MODE == kZero) {
                    if (lane == first) {
#pragma unroll
                        for (int k = 0; k < K; ++k) Mp[k] = Ip[k] = Dp[k] = zero2();
                        gW = zero2();
                    }
                }
                if constexpr (MODE == kReset || CHK) {
                    if (CHK ? (code & kColFirst) != 0 : lane == first) {
                        if (CHK) ++hap;
                        const float init = CHK ? __ldg(B.hap_init_f + hap) : h_init;
                        const float2 X = make_float2(init, rb >= 0 ? init : 0.f);
                        // dummy rows (global slot < pad) hold the row-0 value X in D^; a pad may reach past
                        // strip 0 for the shorter read of a pair
                        const int slot0 = strip * S + lane * K;
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            Mp[k] = Ip[k] = zero2();
                            Dp[k] = make_float2((slot0 + k < task.pad_a) ? X.x : 0.f, (slot0 + k < task.pad_b) ? X.y : 0.f);
                        }
                        const float2 gD = make_float2((slot0 - 1 < task.pad_a) ? X.x : 0.f,
                                                      (slot0 - 1 < task.pad_b) ? X.y : 0.f);
                        gW = mul2(cc[0], gD);
                        if (lane == 0 && strip == 0) w0 = mul2(cc[0], X);
                    }
                }
                if (!(MULTI && strip > 0) && lane == 0) gW = w0;
                const float4 *pri4 = prior_tbl4 + (code & 7u) * 32;
                float2 prs[2 * KP];
#pragma unroll
                for (int kk = 0; kk < KP; ++kk) {
                    const float4 v = pri4[kk * kBases * 32];
                    prs[2 * kk] = make_float2(v.x, v.y);
                    prs[2 * kk + 1] = make_float2(v.z, v.w);
                }
                // pass 1 (bottom-up so the row above is still the previous column): M and D^.  Row k's D~ stands next to
                // the inner sum of row k + 1, which reads the same D~ and M~: three 64-bit operands are more than the
                // register file gives an FFMA2 in its two cycles, and neighbours that share two can reuse them.
#pragma unroll
                for (int k = K - 1; k >= 0; --k) {
                    float2 inner = zero2();
                    if (k + 1 < K) inner = fma2(Dp[k], cc[k + 1], Mp[k]);
                    Dp[k] = fma2(Dp[k], cdd[k], Mp[k]);
                    if (k + 1 < K) Mp[k + 1] = mul2(prs[k + 1], fma2(Ip[k], cb[k + 1], inner));
                }
                Mp[0] = mul2(prs[0], gW);
                // pass 2 (top-down): I~ from the row above at this column; row 0's comes from the lane above
                Ip[0] = uV;
#pragma unroll
                for (int k = 1; k < K; ++k) Ip[k] = fma2(Ip[k - 1], ce[k], Mp[k - 1]);
                // hand the lane below its row 0's I~ at this column and M~ inner sum for the next
                sV = fma2(Ip[K - 1], e0n, Mp[K - 1]);
                sW = fma2(Ip[K - 1], b0n, fma2(Dp[K - 1], c0n, Mp[K - 1]));
                if (last_strip) {
                    if constexpr (CHK) {
                        if (lane == 31 && (code & kColLast)) emit(hap);
                    }
                } else if (MULTI && lane == 31 && s >= 62) {  // (its columns: 0 .. ncols - 1)
                    scratch[c] = make_float4(sV.x, sV.y, sW.x, sW.y);
                }
            };
            // haplotype boundaries of this task: columns hb(j) = hap_off[hap_begin + j] - col0, hb(n) = ncols
            const int64_t *hoff = B.hap_off + task.hap_begin;
            const int nh_task = task.hap_end - task.hap_begin;
            using Plain = std::integral_constant<int, kPlain>;
            using Reset = std::integral_constant<int, kReset>;
            using Zero = std::integral_constant<int, kZero>;
            int s = 0;
            if constexpr (MIXED) {
                // as below for the haplotypes of 63 columns or more; from the boundary of a shorter one on, events of several
                // boundaries overlap, and the steps are checked until those of the next long haplotype's are over
                const int dummies = max(task.pad_a, rb >= 0 ? task.pad_b : 0) - strip * S;  // on top of this strip
                const int n_reset = dummies >= 0 ? min(30, dummies / K + 1) : 0;  // lanes with or right below dummy rows
                bool last_long = false;
                for (int j = 0; j < nh_task;) {  // s: haplotype j's first column
                    int end = (int)(hoff[j + 1] - col0);
                    last_long = end - s >= kShortHapCols;
                    if (last_long) {
                        const float init = __ldg(B.hap_init_f + task.hap_begin + j);
                        int l = 0;
#pragma unroll 1
                        for (; l < n_reset; ++l, s += 2) {
                            refill(s);
                            step(s, Reset{}, l, init);
                            refill(s + 1);
                            step(s + 1, Plain{}, 0, 0.f);
                        }
#pragma unroll 1
                        for (; l < 30; ++l, s += 2) {
                            refill(s);
                            step(s, Zero{}, l, 0.f);
                            refill(s + 1);
                            step(s + 1, Plain{}, 0, 0.f);
                        }
                        refill(s);
                        step(s, Reset{}, 30, init);
                        refill(s + 1);
                        step(s + 1, Plain{}, 0, 0.f);
                        if (j > 0 && last_strip && lane == 31) emit(task.hap_begin + j - 1);
                        refill(s + 2);
                        step(s + 2, Reset{}, 31, init);
                        s += 3;
                        ++j;
                    } else {
                        hap = task.hap_begin + j - 1;
                        int stop = nsteps;
                        for (int begin = s; ++j < nh_task;) {  // haplotype j - 1, from column begin to end, is short
                            begin = end;
                            end = (int)(hoff[j + 1] - col0);
                            if (end - begin >= kShortHapCols) {
                                stop = begin + kShortHapCols;
                                last_long = true;
                                ++j;
                                break;
                            }
                        }
#pragma unroll 2
                        for (; s < stop; ++s) {
                            refill(s);
                            step(s, std::integral_constant<int, kCheck>{}, 0, 0.f);
                        }
                    }
                    const int until = j < nh_task ? end : nsteps;
                    while (s < until) {
                        refill(s);
                        const int stop = MULTI && strip > 0 ? min(until, (s | 31) + 1) : until;
                        // unrolled: the scheduler interleaves one step's I~ chain and shuffles with the following steps' M~
                        // and D~ (16 measured best of 2-32; with the strip boundary 8 of 4, 8 and 16)
                        constexpr int kUnroll = MULTI ? 8 : 16;
#pragma unroll kUnroll
                        for (; s < stop; ++s) step(s, Plain{}, 0, 0.f);
                    }
                }
                if (last_long && last_strip && lane == 31) emit(task.hap_end - 1);
            } else if (long_haps) {
                // Haplotypes of 63 columns or more: at a boundary at column hb, lane l starts the next haplotype at step
                // hb + 2 l and lane 31 ends the previous one at step hb + 61, so which steps have events, and for which
                // lane, is known without looking at a column code, and every other step between two starts is plain.
                // With every step of these 63 checked against the column codes a boundary cost as much as 53 plain
                // steps (FP32 pass over haplotypes of 400 against reads of 254 bases: 4,534 GCUPS, this way 5,088; over haplotypes
                // of 3,200: 5,074).
                const int dummies = max(task.pad_a, rb >= 0 ? task.pad_b : 0) - strip * S;  // on top of this strip
                const int n_reset = dummies >= 0 ? min(30, dummies / K + 1) : 0;  // lanes with or right below dummy rows
                for (int j = 0; j <= nh_task; ++j) {
                    const int until = j < nh_task ? (int)(hoff[j] - col0) : nsteps;
                    while (s < until) {
                        refill(s);
                        const int stop = MULTI && strip > 0 ? min(until, (s | 31) + 1) : until;
                        // unrolled: the scheduler interleaves one step's I~ chain and shuffles with the following steps' M~
                        // and D~ (16 measured best of 2-32; with the strip boundary 8 of 4, 8 and 16)
                        constexpr int kUnroll = MULTI ? 8 : 16;
#pragma unroll kUnroll
                        for (; s < stop; ++s) step(s, Plain{}, 0, 0.f);
                    }
                    if (j == nh_task) break;
                    const float init = __ldg(B.hap_init_f + task.hap_begin + j);
                    int l = 0;
#pragma unroll 1
                    for (; l < n_reset; ++l, s += 2) {
                        refill(s);
                        step(s, Reset{}, l, init);
                        refill(s + 1);
                        step(s + 1, Plain{}, 0, 0.f);
                    }
#pragma unroll 1
                    for (; l < 30; ++l, s += 2) {
                        refill(s);
                        step(s, Zero{}, l, 0.f);
                        refill(s + 1);
                        step(s + 1, Plain{}, 0, 0.f);
                    }
                    refill(s);
                    step(s, Reset{}, 30, init);
                    refill(s + 1);
                    step(s + 1, Plain{}, 0, 0.f);
                    if (j > 0 && last_strip && lane == 31) emit(task.hap_begin + j - 1);
                    refill(s + 2);
                    step(s + 2, Reset{}, 31, init);
                    s += 3;
                }
                if (last_strip && lane == 31) emit(task.hap_end - 1);
            } else {  // most are shorter
#pragma unroll 2
                for (; s < nsteps; ++s) {
                    refill(s);
                    step(s, std::integral_constant<int, kCheck>{}, 0, 0.f);
                }
            }
            if (MULTI) __syncwarp();
        }
    }
}

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
static size_t fp32_smem_bytes(int k, int block, bool multi) {
    return (size_t)(block / 32) * (((k + 1) / 2) * kBases * 32 + (multi ? 64 : 0)) * sizeof(float4);
}

template <int K, bool MULTI, bool MIXED>
static int launch_fp32_k(const DevTables &t, const DevBatch &b, int grid, int block, cudaStream_t s) {
    const size_t smem = fp32_smem_bytes(K, block, MULTI);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(fp32_bucket_kernel<K, MULTI, MIXED>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    fp32_bucket_kernel<K, MULTI, MIXED><<<grid, block, smem, s>>>(t, b);
    return (int)cudaGetLastError();
}

// f(rows per lane, several strips, mixed haplotypes), as integral constants, of a bucket key
template <typename F>
static int with_bucket(int key, F f) {
    switch (bucket_rows(key)) {
#define GHMM_CASE(KK)                                                                                                     \
    case KK: {                                                                                                            \
        using K = std::integral_constant<int, KK>;                                                                        \
        if (key & kBucketMulti)                                                                                           \
            return bucket_mixed(key) ? f(K{}, std::true_type{}, std::true_type{}) : f(K{}, std::true_type{}, std::false_type{}); \
        return bucket_mixed(key) ? f(K{}, std::false_type{}, std::true_type{}) : f(K{}, std::false_type{}, std::false_type{}); \
    }
        GHMM_CASE(2)
        GHMM_CASE(3)
        GHMM_CASE(4)
        GHMM_CASE(5)
        GHMM_CASE(6)
        GHMM_CASE(7)
        GHMM_CASE(8)
#undef GHMM_CASE
        default:
            return (int)cudaErrorInvalidValue;
    }
}

int launch_fp32_bucket(const DevTables &t, const DevBatch &b, int key, int grid, int block, cudaStream_t s) {
    return with_bucket(key, [&](auto k, auto multi, auto mixed) {
        return launch_fp32_k<k.value, multi.value, mixed.value>(t, b, grid, block, s);
    });
}

int fp32_kernel_occupancy(int key, int block, int *blocks_per_sm) {
    return with_bucket(key, [&](auto k, auto multi, auto mixed) {
        return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            blocks_per_sm, fp32_bucket_kernel<k.value, multi.value, mixed.value>, block,
            fp32_smem_bytes(k.value, block, multi.value));
    });
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
