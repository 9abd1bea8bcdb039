// fp64.cu -- the FP64 wavefront: reruns of FP32 underflows, pairs routed to FP64, and double-precision mode, in two
// tiers of one kernel template.  (Recurrence and citations: kernels.cu.)
//
// RESCALED (queue 1: host-routed pairs and FP32 underflows): the FP32 kernel's rescaled recurrence in FP64,
// 5 DP operations per cell instead of 8 (the FP64 pipe runs at 1/64 of the FP32 rate on this part):
//    M~ = prior * fma(I~_diag, b_i, fma(D~_diag, c_i, M~_diag)),  I~ = fma(I~_up, e_i, M~_up),
//    D~ = fma(D~_left, DD_i, M~_left),  sum over the haplotype of M~_R + (MI_R / MM_R) I~_R.
// The scale is S' = 2^960 instead of 2^1020 (headroom for I~ and D~, which carry 1 / MI and 1 / MD), and the
// initial condition is divided by 2^round(la), la = log2 a_R = sum of -log2 MM_i, so that the last row sits at
// scale S' like the unscaled recurrence.  Along every contributing path the rescaled states stay above the
// final sum's magnitude, so a result of log10 L >= kRescaledFloor (well inside the FP64 range at S') is as
// accurate as the unscaled recurrence; lower or non-finite results go to queue 2.
//
// EXACT (queue 2: those, and reads the host marks, e.g. matchToMatch ~ 0): the unscaled recurrence with the
// reference's 2^1020 initial condition, so it underflows exactly where LoglessPairHMM does.
//
// What bounds it: the FP64 pipe, and that pipe is one per SM sub-partition: a warp's DFMA takes 64 cycles whether or
// not the other three sub-partitions work (register loop: 0.156 Tops/s with one warp per SM at any instruction-level
// parallelism, 0.625 with four).  Hence:
//  * Everything but DP operations is free (64 issue slots per DP operation), and every DP operation counts.  A DMUL or
//    DADD costs 19 cycles an SM where a DFMA costs 16, also a DFMA that the compiler can turn into one, so products
//    and sums are DFMAs with a zero (or one) that only run time knows: the same roundings.  The last row is summed by
//    all lanes once per 16 columns instead of by one lane in every column (two of 22 DP operations a step before).
//  * Padding is work: a read's rows are split into strips of 32, 64, 96 or 128 rows that cover ceil(R / 32) * 32 rows
//    instead of whole strips of 128 (reads of 100-250 bases: 191 rows on average instead of 232).
//  * The wavefront's fill is work too: 31 of some 430 steps of a short read's strip.  A warp therefore takes a run of up to
//    four neighbouring queue entries of one read and consecutive haplotypes (as routed pairs and double-precision mode
//    queue them) as one stream of columns, in which each lane resets its state at a haplotype's first column.
//  * A pair on one warp uses a quarter of one SM.  Jobs are therefore either a pair per warp, its strips one after the
//    other, or a pair per block: the strips go round the block's four warps, each strip 48 columns behind the one above
//    it, in lockstep phases of 16 columns.
// Measured against one pair per warp in strips of 128 rows (one GB300): 537 reads of 800-2,000 bases x haplotypes of
// 1,500-3,000 (1.6e10 cells) 214 -> 158 ms, 103 of at most 125 GCUPS; 37,978 pairs of 100-250 bases (2.6e9 cells) all in
// FP64 36.3 -> 27.2 ms; the 5 reruns of a region of 2,000 reads 0.85 -> 0.34 ms; 48 reruns of 260-600 bases x 800
// 3.6 -> 1.1 ms.  Runs of haplotypes on top: the 37,978 pairs 27.2 -> 26.0 ms.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/ghmm.h"
#include "ghmm_internal.h"

namespace ghmm {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarps64 = 4;    // warps per block
constexpr int kPhase = 16;     // columns (steps) of one phase
constexpr int kStripLag = 3;   // phases a strip stays behind the strip above it: column c of the row above is written at
                               // that strip's step c + 31, i.e. by the end of phase c / 16 + 2 at the latest
constexpr double kLog10Scale64R = 288.9887958374219;   // log10(2^960)
constexpr double kLog10Scale64 = 307.0505955772608;    // log10(2^1020)
constexpr double kRescaledFloor = GHMM_FP64_RESCALED_FLOOR;

// x * y and x + y at the DFMA rate; zero and one are kernel arguments, unknown to the compiler.  Every product here is
// >= 0, so adding zero keeps its bits.
struct Unit {
    double zero, one;
};
__device__ __forceinline__ double mul64(double x, double y, Unit u) { return fma(x, y, u.zero); }
__device__ __forceinline__ double add64(double x, double y, Unit u) { return fma(x, u.one, y); }

// The read of a job and its haplotypes: n consecutive ones, n > 1 in a warp's runs only.
struct Pair64 {
    int64_t roff, out_index;  // of the first haplotype's result; the others' follow
    const uint8_t *hb;
    int read, hap, n, R, H;   // H: columns of all n haplotypes
    int blocks32;             // rows / 32, rounded up: the rows of all strips
    int pad;                  // dummy rows on top of strip 0 (0..31); they hold the row-0 boundary
    double la;
};

// What lanes look up when they start a haplotype, in shared memory per warp: row-0 values and end columns.
constexpr int kRun64 = kFp64Run;
struct Run64 {
    double init[kRun64];
    int end[kRun64];
};

__device__ __forceinline__ Pair64 load_pair(const DevBatch &B, PairRef pr, int n = 1) {
    Pair64 P;
    P.read = pr.read;
    P.hap = pr.hap;
    P.n = n;
    P.roff = B.read_off[pr.read];
    P.R = (int)(B.read_off[pr.read + 1] - P.roff);
    const int64_t hoff = B.hap_off[pr.hap];
    P.H = (int)(B.hap_off[pr.hap + n] - hoff);
    P.hb = B.hap_bases + hoff;
    const int region = B.read_region[pr.read];
    const int64_t nh = B.region_hap_off[region + 1] - B.region_hap_off[region];
    P.out_index = B.out_off[region] + (int64_t)(pr.read - B.region_read_off[region]) * nh +
                  (pr.hap - B.region_hap_off[region]);
    P.blocks32 = (P.R + 31) / 32;
    P.pad = P.blocks32 * 32 - P.R;
    P.la = 0.0;
    return P;
}

// One strip of K <= 4 rows per lane: coefficients and running states of this lane's rows.
template <bool RESCALED>
struct Strip64 {
    double pm[4], pe[4];
    double c1[4], c2[4], c3[4], c4[4];  // RESCALED: b, c, e, unused; exact: MM, IM, MI, II
    double c5[4];                       // exact: MD
    double dd[4];                       // DD (1 in dummy rows, whose D stays at the row-0 value)
    double M[4], I[4], D[4];
    uint32_t base[4];
    double gM, gI, gD;     // row above the lane's first row, previous column
    double nxM, nxI, nxD;  // lane 0 below the first strip: the row above at the next column
    double init;           // row-0 value of the haplotype the lane is in
    int start, hap;        // first column and ordinal of the haplotype the lane enters next
    int row0, k;           // first row (slot) of the strip, rows per lane
    bool first, last;
};

// Strip `strip` of n strips that share the pair's 32-row blocks as evenly as they go, the larger ones first.
template <bool RESCALED>
__device__ __forceinline__ void strip_begin(const DevTables &T, const DevBatch &B, const Pair64 &P, int strip, int n,
                                            double init, const double *above, Strip64<RESCALED> &S, int lane) {
    const int even = P.blocks32 / n, more = P.blocks32 - even * n;
    S.k = even + (strip < more ? 1 : 0);
    S.row0 = 32 * (strip * even + min(strip, more));
    S.first = strip == 0;
    S.last = strip == n - 1;
    S.start = S.hap = 0;
    S.init = init;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int p = S.row0 + lane * S.k + k - P.pad;
        S.pm[k] = S.pe[k] = S.c1[k] = S.c2[k] = S.c3[k] = S.c4[k] = S.c5[k] = 0.0;
        S.dd[k] = 1.0;
        S.base[k] = 0x100u;  // matches nothing
        if (k < S.k && p >= 0) {
            const uint8_t base = B.bases[P.roff + p], q = B.quals[P.roff + p];
            const uint8_t ins = B.ins[P.roff + p], del = B.dels[P.roff + p], gcp = B.gcp[P.roff + p];
            S.pm[k] = __ldg(T.prob_d + q);
            S.pe[k] = base == 'N' ? S.pm[k] : __ldg(T.err3_d + q);
            S.base[k] = base;
            const double mm = __ldg(T.m2m_d + ins * 128 + del), im = __ldg(T.prob_d + gcp);
            const double mi = __ldg(T.err_d + ins), ii = __ldg(T.err_d + gcp), md = __ldg(T.err_d + del);
            S.dd[k] = ii;
            if (RESCALED) {
                double mm_p = 1.0, mi_p = 1.0, md_p = 1.0;
                if (p > 0) {
                    const uint8_t ins_p = B.ins[P.roff + p - 1], del_p = B.dels[P.roff + p - 1];
                    mm_p = __ldg(T.m2m_d + ins_p * 128 + del_p);
                    mi_p = __ldg(T.err_d + ins_p);
                    md_p = __ldg(T.err_d + del_p);
                }
                S.c1[k] = im * mi_p / (mm * mm_p);
                S.c2[k] = im * md_p / mm;
                S.c3[k] = p > 0 ? ii * mi_p / (mi * mm_p) : 0.0;
            } else {
                S.c1[k] = mm;
                S.c2[k] = im;
                S.c3[k] = mi;
                S.c4[k] = ii;
                S.c5[k] = md;
            }
        }
    }
    if (!S.first && lane == 0) {
        S.nxM = above[0];
        S.nxI = above[1];
        S.nxD = above[2];
    }
}

// Steps [s0, s1) of a strip of K rows per lane: at step s lane l computes column s - l.  The last row of a strip goes
// to `below` for the next strip; the pair's last row goes to rowM / rowI, 16 steps at a time.
template <int K, bool RESCALED>
__device__ __forceinline__ void strip_steps(const Pair64 &P, const Run64 &run, Strip64<RESCALED> &S, int s0, int s1,
                                            const double *above, double *below, double *rowM, double *rowI, Unit u,
                                            int lane) {
    for (int s = s0; s < s1; ++s) {
        const int c = s - lane;
        const bool valid = c >= 0 && c < P.H;
        const uint32_t y = valid ? (uint32_t)__ldg(P.hb + c) : 0x200u;
        const bool yn = (y == 'N');
        const bool enter = c == S.start;  // a haplotype's column-0 boundary (lanes compute ahead of their first column)
        if (P.n > 1 && enter) {
            S.init = run.init[S.hap];
            S.start = run.end[S.hap];
            S.hap = min(S.hap + 1, P.n - 1);  // (a lane past the last column resets a state that nothing reads)
        }
        double uM = __shfl_up_sync(kFull, S.M[K - 1], 1);  // (the lane below still needs the column before)
        double uI = __shfl_up_sync(kFull, S.I[K - 1], 1);
        double uD = __shfl_up_sync(kFull, S.D[K - 1], 1);
        if (enter) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                S.M[k] = S.I[k] = 0.0;
                S.D[k] = (S.first && lane * K + k < P.pad) ? S.init : 0.0;
            }
            S.gM = S.gI = 0.0;
            S.gD = (S.first && lane * K - 1 < P.pad) ? S.init : 0.0;
        }
        if (lane == 0) {
            if (S.first) {
                uM = 0.0;
                uI = 0.0;
                uD = S.init;
            } else {
                uM = S.nxM;
                uI = S.nxI;
                uD = S.nxD;
                if (c + 1 < P.H) {
                    S.nxM = above[3 * (c + 1) + 0];
                    S.nxI = above[3 * (c + 1) + 1];
                    S.nxD = above[3 * (c + 1) + 2];
                }
            }
        }
#pragma unroll
        for (int k = K - 1; k >= 0; --k) {
            const double dM = k ? S.M[k - 1] : S.gM;
            const double dI = k ? S.I[k - 1] : S.gI;
            const double dD = k ? S.D[k - 1] : S.gD;
            const double prior = (S.base[k] == y || yn) ? S.pm[k] : S.pe[k];
            double Mn, Dn;
            if (RESCALED) {
                Mn = mul64(prior, fma(dI, S.c1[k], fma(dD, S.c2[k], dM)), u);
                Dn = fma(S.D[k], S.dd[k], S.M[k]);
            } else {  // the reference's grouping: prior x (M x MM + (I + D) x IM), so results deep in the
                      // subnormal range round as LoglessPairHMM's do
                Mn = mul64(prior, fma(dM, S.c1[k], mul64(add64(dI, dD, u), S.c2[k], u)), u);
                Dn = fma(S.D[k], S.dd[k], mul64(S.M[k], S.c5[k], u));
            }
            S.M[k] = Mn;
            S.D[k] = Dn;
        }
        double aM = uM, aI = uI;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const double In = RESCALED ? fma(aI, S.c3[k], aM) : fma(aI, S.c4[k], mul64(aM, S.c3[k], u));
            S.I[k] = In;
            aM = S.M[k];
            aI = In;
        }
        S.gM = uM;
        S.gI = uI;
        S.gD = uD;
        if (valid && lane == 31) {
            if (S.last) {
                rowM[s - s0] = S.M[K - 1];
                rowI[s - s0] = S.I[K - 1];
            } else {
                below[3 * c + 0] = S.M[K - 1];
                below[3 * c + 1] = S.I[K - 1];
                below[3 * c + 2] = S.D[K - 1];
            }
        }
    }
}

// The pair's scale (RESCALED): la = log2 a_R and the initial condition divided by 2^round(la); all lanes.  Fills the
// warp's table of its haplotypes.
template <bool RESCALED>
__device__ __forceinline__ void pair_scale(const DevTables &T, const DevBatch &B, Pair64 &P, Run64 &run, double &kappa,
                                           int lane) {
    kappa = 1.0;
    int shift = 0;
    if (RESCALED) {
        double la = 0.0;
        for (int p = lane; p < P.R; p += 32) la += __ldg(T.lm2m64 + B.ins[P.roff + p] * 128 + B.dels[P.roff + p]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) la += __shfl_xor_sync(kFull, la, o);
        P.la = la;
        shift = -60 - (int)rint(la);
        const uint8_t ins = B.ins[P.roff + P.R - 1], del = B.dels[P.roff + P.R - 1];
        kappa = __ldg(T.err_d + ins) / __ldg(T.m2m_d + ins * 128 + del);
    }
    __syncwarp();  // the last job's steps have read the table
    if (lane < P.n) {
        run.init[lane] = scalbn(B.hap_init_d[P.hap + lane], shift);
        run.end[lane] = (int)(B.hap_off[P.hap + lane + 1] - B.hap_off[P.hap]);
    }
    __syncwarp();
}

// The result of haplotype h of the job from the lanes' parts of the sum over its last row.
template <bool RESCALED>
__device__ __forceinline__ void pair_emit(const DevBatch &B, const Pair64 &P, int h, double acc, int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
    if (lane != 0) return;
    if (RESCALED) {
        const double rla = rint(P.la);
        const double v = log10(acc) - kLog10Scale64R - (P.la - rla) * 0.30102999566398120;
        if (v >= kRescaledFloor && v <= 0.0) {
            B.out[P.out_index + h] = v;
        } else {  // too close to the FP64 range at S' (or not finite): the exact tier recomputes it
            const int idx = atomicAdd(&B.counters[4], 1);
            if ((int64_t)idx < B.rerun_capacity)
                B.rerun[B.rerun_capacity + idx] = PairRef{P.read, P.hap + h};
            else
                atomicExch(&B.counters[3], 1);
        }
    } else {
        B.out[P.out_index + h] = log10(acc) - kLog10Scale64;
    }
}

// What a warp keeps of the sums of a job's last row: the haplotype being summed and this lane's part.
struct Sum64 {
    double acc = 0.0;
    int hap = 0;
    int end;  // of that haplotype's columns
};

// Phase r (steps 16 r .. 16 r + 15) of a strip.  After the last strip's, lane l adds the last row's column of step
// 16 r + l, and the results of the haplotypes that end among these columns are stored.
template <bool RESCALED>
__device__ __forceinline__ void strip_phase(const DevBatch &B, const Pair64 &P, const Run64 &run, Strip64<RESCALED> &S, int r,
                                            const double *above, double *below, double *rowM, double *rowI, double kappa,
                                            Sum64 &sum, Unit u, int lane) {
    const int s0 = r * kPhase, s1 = min(s0 + kPhase, P.H + 31);
    switch (S.k) {
        case 1: strip_steps<1, RESCALED>(P, run, S, s0, s1, above, below, rowM, rowI, u, lane); break;
        case 2: strip_steps<2, RESCALED>(P, run, S, s0, s1, above, below, rowM, rowI, u, lane); break;
        case 3: strip_steps<3, RESCALED>(P, run, S, s0, s1, above, below, rowM, rowI, u, lane); break;
        default: strip_steps<4, RESCALED>(P, run, S, s0, s1, above, below, rowM, rowI, u, lane); break;
    }
    if (!S.last) return;
    __syncwarp();
    const int c = s0 + lane - 31;
    double v = 0.0;
    if (s0 + lane < s1 && c >= 0) v = RESCALED ? fma(kappa, rowI[lane], rowM[lane]) : rowM[lane] + rowI[lane];
    __syncwarp();
    int from = s0 - 31;  // columns [from, s1 - 31) are new
    while (sum.end <= s1 - 31) {
        if (c >= from && c < sum.end) sum.acc += v;
        pair_emit<RESCALED>(B, P, sum.hap, sum.acc, lane);
        sum.acc = 0.0;
        from = sum.end;
        sum.end = ++sum.hap < P.n ? run.end[sum.hap] : INT32_MAX;
    }
    if (c >= from && s0 + lane < s1) sum.acc += v;
}

// A read without bases or a haplotype without columns: -inf, as in Java; one beyond the strip scratch: an error.
__device__ __forceinline__ bool pair_skipped(const DevBatch &B, const Pair64 &P, bool writer) {
    if (P.R == 0 || P.H == 0) {
        if (writer)
            for (int h = 0; h < P.n; ++h) B.out[P.out_index + h] = -INFINITY;
        return true;
    }
    if (P.H > B.scratch64_cols && P.blocks32 > 1) {
        if (writer) atomicExch(&B.counters[3], 2);
        return true;
    }
    return false;
}

__device__ __forceinline__ bool long_pair(const DevBatch &B, PairRef pr) {
    return B.read_off[pr.read + 1] - B.read_off[pr.read] >= kFp64SplitRows;
}

// Lists the queue's entries of long reads (their indices, in the queue's order), for batches that have such reads: each
// block those of its part of the queue, behind those that it counts in the parts before (half a millisecond for a million
// entries).  In any order that atomics give, 5,172 pairs of 800-2,000 bases took 161 ms instead of 158.
constexpr int kListThreads = 1024;
template <bool RESCALED>
__global__ void __launch_bounds__(kListThreads) fp64_long_kernel(DevBatch B, int32_t *long_list) {
    __shared__ int warp_count[kListThreads / 32];
    const PairRef *queue = RESCALED ? B.rerun : B.rerun + B.rerun_capacity;
    const int total = min(B.counters[RESCALED ? 1 : 4], (int)B.rerun_capacity);
    const int begin = (int)((int64_t)total * blockIdx.x / gridDim.x);
    const int end = (int)((int64_t)total * (blockIdx.x + 1) / gridDim.x);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int at = 0;
    for (int base = 0; base < begin; base += kListThreads) {
        const int i = base + (int)threadIdx.x;
        at += __syncthreads_count(i < begin && long_pair(B, queue[i]));
    }
    for (int base = begin; base < end; base += kListThreads) {
        const int i = base + (int)threadIdx.x;
        const bool found = i < end && long_pair(B, queue[i]);
        const unsigned mine = __ballot_sync(kFull, found);
        if (lane == 0) warp_count[warp] = __popc(mine);
        const int here = __syncthreads_count(found);
        int slot = at + __popc(mine & ((1u << lane) - 1u));
        for (int w = 0; w < warp; ++w) slot += warp_count[w];
        if (found) long_list[slot] = i;
        at += here;
        __syncthreads();  // every warp has read the counts
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) B.counters[kCounterFp64Long + (RESCALED ? 0 : 2)] = at;
}

// The entries of a long list, a pair or run per warp (LONG: but for the long reads'): drawn several at a time while many a
// warp are left, one by one towards the end.
template <bool RESCALED, bool LONG>
__device__ __forceinline__ void pairs_by_warp(const DevTables &T, const DevBatch &B, const PairRef *queue, int total,
                                              int *cursor, int warps, Run64 &run, double *mine, double *rowM,
                                              double *rowI, Unit u, int lane,
                                              Strip64<RESCALED> &S, double &kappa) {
    for (;;) {
        int t0 = 0, draw = 1;
        if (lane == 0) {
            const int left = total - *reinterpret_cast<volatile int *>(cursor);
            draw = max(1, min(kRun64, left / (2 * warps)));
            t0 = atomicAdd(cursor, draw);
        }
        t0 = __shfl_sync(kFull, t0, 0);
        draw = __shfl_sync(kFull, draw, 0);
        if (t0 >= total) break;
        const int t1 = min(t0 + draw, total);
        for (int t = t0; t < t1;) {
            const PairRef pr = queue[t];
            if (LONG && long_pair(B, pr)) {
                ++t;
                continue;
            }
            // a run: the same read, the haplotype after the last one's, no empty ones, within the strip scratch
            int n = 1;
            const int64_t h0 = B.hap_off[pr.hap];
            int64_t end = B.hap_off[pr.hap + 1];
            while (t + n < t1 && end > h0) {
                const PairRef next = queue[t + n];
                if (next.read != pr.read || next.hap != pr.hap + n) break;
                const int64_t e = B.hap_off[next.hap + 1];
                if (e == end || e - h0 > B.scratch64_cols) break;
                end = e;
                ++n;
            }
            t += n;
            Pair64 P = load_pair(B, pr, n);
            if (pair_skipped(B, P, lane == 0)) continue;
            pair_scale<RESCALED>(T, B, P, run, kappa, lane);
            const int strips = (P.blocks32 + 3) / 4, phases = (P.H + 31 + kPhase - 1) / kPhase;
            Sum64 sum;
            sum.end = run.end[0];
            for (int strip = 0; strip < strips; ++strip) {
                __syncwarp();  // the strip above has written its last row
                strip_begin<RESCALED>(T, B, P, strip, strips, run.init[0], mine, S, lane);
                for (int r = 0; r < phases; ++r)
                    strip_phase<RESCALED>(B, P, run, S, r, mine, mine, rowM, rowI, kappa, sum, u, lane);
            }
        }
    }
}

// Launched with full grids; queue lengths are device counters, so the choice between a pair per warp and a pair per
// block is made here.  A pair per block when the list is shorter than the grid's warps (each pair then runs on four
// sub-partitions).  Of longer lists, the pairs of long reads, which go first (LONG, for batches that have such reads:
// long_list names their entries): a pair's time on one warp, 15 ms at 1,400 x 2,250 bases, is what the last pairs would
// otherwise take.  A pair per warp for the others: in a block they idle warps in the strips' lag and, having fewer strips
// than warps, altogether (10,240 pairs of 20, 100 and 250 x 300 bases beside one of 481 x 600: 1.11, 3.74 and 7.42 ms; all
// of them a pair per block 3.05, 5.57 and 8.98).
template <bool RESCALED, bool LONG>
__global__ void __launch_bounds__(32 * kWarps64, 3) fp64_queue_kernel(DevTables T, DevBatch B, const int32_t *long_list,
                                                                      Unit u) {
    __shared__ double row_sum[kWarps64][2][kPhase];
    __shared__ Run64 runs[kWarps64];
    __shared__ int job;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const PairRef *queue = RESCALED ? B.rerun : B.rerun + B.rerun_capacity;
    const int total = min(B.counters[RESCALED ? 1 : 4], (int)B.rerun_capacity);
    int *const cursor = &B.counters[RESCALED ? 2 : 5];
    double *const block_scratch = B.scratch64 + (int64_t)blockIdx.x * kWarps64 * B.scratch64_cols * 3;
    double *const mine = block_scratch + (int64_t)warp * B.scratch64_cols * 3;
    double *const rowM = row_sum[warp][0], *const rowI = row_sum[warp][1];
    Run64 &run = runs[warp];
    Strip64<RESCALED> S;
    double kappa;
    const int warps = (int)gridDim.x * kWarps64;
    if (!LONG && total > warps) {
        pairs_by_warp<RESCALED, LONG>(T, B, queue, total, cursor, warps, run, mine, rowM, rowI, u, lane, S, kappa);
        return;
    }
    // a pair per block: the whole queue, or of a long one the listed entries
    const bool listed = LONG && total > warps;
    int *const counters = &B.counters[kCounterFp64Long + (RESCALED ? 0 : 2)];
    const int n_pairs = listed ? counters[0] : total;
    int *const next_pair = listed ? counters + 1 : cursor;
    const double *const above = block_scratch + (int64_t)((warp + kWarps64 - 1) % kWarps64) * B.scratch64_cols * 3;
    for (bool first = true;;) {
        int t = blockIdx.x;
        if (!first) {
            __syncthreads();  // every warp has read the previous job
            if (threadIdx.x == 0) job = (int)gridDim.x + atomicAdd(next_pair, 1);
            __syncthreads();
            t = job;
        }
        first = false;
        if (t >= n_pairs) break;
        Pair64 P = load_pair(B, queue[listed ? long_list[t] : t]);
        if (pair_skipped(B, P, threadIdx.x == 0)) continue;
        pair_scale<RESCALED>(T, B, P, run, kappa, lane);
        // strips of at most 128 rows, a multiple of four of them where the rows allow; strip s runs on warp s % 4 from
        // phase start(s) = (s / 4) round + (s % 4) lag on, round being a strip's phases and long enough for the strip
        // that wraps round to warp 0 to stay behind the one above it on warp 3
        const int n = min(((P.blocks32 + 3) / 4 + 3) / 4 * 4, P.blocks32);
        const int phases = (P.H + 31 + kPhase - 1) / kPhase;
        const int round = max(phases, kStripLag * kWarps64);
        const int end = (n - 1) / kWarps64 * round + (n - 1) % kWarps64 * kStripLag + phases;
        int strip = warp, start = warp * kStripLag;
        Sum64 sum;
        sum.end = P.H;
        for (int p = 0; p < end; ++p) {
            if (strip < n && p >= start) {
                if (p == start) strip_begin<RESCALED>(T, B, P, strip, n, run.init[0], above, S, lane);
                strip_phase<RESCALED>(B, P, run, S, p - start, above, mine, rowM, rowI, kappa, sum, u, lane);
                if (p - start == phases - 1) {
                    strip += kWarps64;
                    start += round;
                }
            }
            __syncthreads();
        }
    }
    if (listed) pairs_by_warp<RESCALED, LONG>(T, B, queue, total, cursor, warps, run, mine, rowM, rowI, u, lane, S, kappa);
}

}  // namespace

int launch_fp64_queue(const DevTables &t, const DevBatch &b, int32_t *long_list, int grid, int sm_count, cudaStream_t s) {
    const Unit u{0.0, 1.0};
    if (long_list) {
        fp64_long_kernel<true><<<sm_count, kListThreads, 0, s>>>(b, long_list);
        fp64_queue_kernel<true, true><<<grid, 32 * kWarps64, 0, s>>>(t, b, long_list, u);
        fp64_long_kernel<false><<<sm_count, kListThreads, 0, s>>>(b, long_list);
        fp64_queue_kernel<false, true><<<grid, 32 * kWarps64, 0, s>>>(t, b, long_list, u);
    } else {
        fp64_queue_kernel<true, false><<<grid, 32 * kWarps64, 0, s>>>(t, b, nullptr, u);
        fp64_queue_kernel<false, false><<<grid, 32 * kWarps64, 0, s>>>(t, b, nullptr, u);
    }
    return (int)cudaGetLastError();
}

int fp64_kernel_occupancy(int *blocks_per_sm) {
    // both tiers run on the same grid and scratch: the smallest occupancy of the forms
    const void *fns[] = {(const void *)fp64_queue_kernel<true, false>, (const void *)fp64_queue_kernel<false, false>,
                         (const void *)fp64_queue_kernel<true, true>, (const void *)fp64_queue_kernel<false, true>};
    cudaError_t e = cudaSuccess;
    *blocks_per_sm = INT32_MAX;
    for (const void *fn : fns) {
        int n = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, 32 * kWarps64, 0);
        *blocks_per_sm = n < *blocks_per_sm ? n : *blocks_per_sm;
    }
    return (int)e;
}

}  // namespace ghmm
