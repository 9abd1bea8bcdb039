// fp32_bucket.cuh -- the batched FP32 forward's kernel (described in kernels.cu), for the tasks of one kind: those of mixed
// haplotypes (kBucketMixed) or the others.  A translation unit defines kMixedTasks before it includes this: with both forms
// in one kernel, or chosen by a template argument, the compiler's code for the usual tasks is 1 to 4 % slower.  Internal
// linkage: each translation unit gets its own kernels.
#pragma once
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

// Blocks of 128 threads the FP32 kernel asks ptxas to fit per SM (register budget 65536 / (128 * n)).  K <= 5 fits
// four without spilling (126 registers at K = 5: 0.4 % faster than three); K = 6 and 7 at four spill a little and
// ran 1-2 % slower, K = 8 spills 600 bytes.
template <int K>
struct Fp32MinBlocks {
    static constexpr int value = K >= 6 ? 3 : 4;
};

// The bucket's task range and cursor live in device memory (B.bucket_info, B.counters), so the launch
// arguments do not depend on the batch and a captured CUDA graph can be replayed for every batch.
template <int K, bool MULTI>
__global__ void __launch_bounds__(128, Fp32MinBlocks<K>::value) fp32_bucket_kernel(DevTables T, DevBatch B) {
    constexpr int KEY = K + (kMixedTasks ? kBucketMixed : 0) + (MULTI ? kBucketMulti : 0);
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
        if constexpr (!kMixedTasks) {
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
            if constexpr (kMixedTasks) {
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

size_t fp32_smem_bytes(int k, int block, bool multi) {
    return (size_t)(block / 32) * (((k + 1) / 2) * kBases * 32 + (multi ? 64 : 0)) * sizeof(float4);
}

template <int K, bool MULTI>
int launch_fp32_k(const DevTables &t, const DevBatch &b, int grid, int block, cudaStream_t s) {
    const size_t smem = fp32_smem_bytes(K, block, MULTI);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(fp32_bucket_kernel<K, MULTI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    fp32_bucket_kernel<K, MULTI><<<grid, block, smem, s>>>(t, b);
    return (int)cudaGetLastError();
}

// f(rows per lane, several strips), as integral constants, of a bucket key
template <typename F>
int with_bucket(int key, F f) {
    switch (bucket_rows(key)) {
#define GHMM_CASE(KK)                                                            \
    case KK:                                                                     \
        return key & kBucketMulti ? f(std::integral_constant<int, KK>{}, std::true_type{}) \
                                  : f(std::integral_constant<int, KK>{}, std::false_type{});
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

int launch_fp32_form(const DevTables &t, const DevBatch &b, int key, int grid, int block, cudaStream_t s) {
    return with_bucket(key, [&](auto k, auto multi) {
        return launch_fp32_k<decltype(k)::value, decltype(multi)::value>(t, b, grid, block, s);
    });
}

int fp32_form_occupancy(int key, int block, int *blocks_per_sm) {
    return with_bucket(key, [&](auto k, auto multi) {
        constexpr int K = decltype(k)::value;
        constexpr bool kMulti = decltype(multi)::value;
        return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fp32_bucket_kernel<K, kMulti>, block,
                                                                  fp32_smem_bytes(K, block, kMulti));
    });
}

}  // namespace
}  // namespace ghmm
