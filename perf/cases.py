"""Performance cases of the read-likelihood library: the calls that HaplotypeCaller / Mutect2 hosts make.

A host program keeps one engine (``Engine``, or the PairHMM plugin object) for its lifetime and hands it new
regions on every call, in host memory, and takes the results in host memory; a program that goes on working on a
batch (normalisation, realignment) holds a ``Batch``.  The cases run those calls whole.  Inputs come from the
repository's generator (region, read and haplotype distributions of ``include/ghmm_synth.h``) or, for one region
of given sizes, from ``_one_region`` below with the same error and quality model.

``exact`` restates the recurrences in 64-bit torch over anti-diagonals; it uses none of the library's code.
"""
import math

import numpy as np
import torch

from gatk_gb300 import calibration, smithwaterman, workload
from gatk_gb300.pairhmm import CudaLoglessPairHMM, Engine, PairHMMNativeArguments

MEAN_READS, MEAN_HAPS, MEAN_HAP_LEN, MEAN_READ_LEN = 88.8, 17.0, 400.0, 175.0  # of its lognormal / uniform draws
_ENGINES = {}           # what a host process keeps: one engine per precision, one plugin object, one queue


def listed():
    return [
        # One JNI call of HaplotypeCaller: one region's reads against its haplotypes.  Latency counts.
        {"name": "one_region_call", "kind": "plugin", "reads": 64, "haps": 8, "read_lo": 150, "read_hi": 150,
         "hap_len": 300},
        # A high-depth region (2,000 reads x 64 haplotypes), called by itself.
        {"name": "deep_region", "kind": "region", "reads": 2000, "haps": 64, "read_lo": 100, "read_hi": 250,
         "hap_len": 450},
        # Reads longer than one strip of the FP32 wavefront (merged pairs, long amplicons).
        {"name": "long_read_region", "kind": "region", "reads": 600, "haps": 24, "read_lo": 260, "read_hi": 600,
         "hap_len": 800},
        # A batch kept on the device and evaluated again (forward and results).
        {"name": "batch_forward", "kind": "batch", "regions": 600},
        # The batched call at its largest: thousands of regions from host memory in one synchronous call.
        {"name": "regions_large", "kind": "compute", "regions": 6000},
        # Regions pushed one at a time, as HaplotypeCaller produces them; 5 % are 2,000 reads x 64 haplotypes.
        {"name": "region_stream", "kind": "stream", "regions": 200},
        # Long reads of low quality (800-2,000 bases): nearly every pair needs FP64.
        {"name": "long_pairs", "kind": "long", "regions": 16},
        # useDoublePrecision: every pair in FP64.
        {"name": "double_precision", "kind": "double", "regions": 40},
        # One step of the gap-penalty calibration: log10 likelihoods and the gradient of the table.
        {"name": "calibration_step", "kind": "calib", "regions": 512},
        # Partially determined haplotypes (the DRAGEN-GATK mode).
        {"name": "pd_regions", "kind": "pd", "regions": 300},
        # The whole step from raw reads: preparation, likelihoods, normalisation and filter, realignment.
        {"name": "raw_step", "kind": "raw", "regions": 150, "imputation": "dragstr"},
        # Reads of a held batch realigned to their best haplotypes (Smith-Waterman).
        {"name": "realign", "kind": "realign", "regions": 600},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plugin", "region", "region", "batch", "compute", "compute", "stream", "long", "double", "calib",
                       "pd", "raw", "realign"])
    if kind in ("plugin", "region"):
        lo = _log_int(rng, 30, 400)
        hi = lo + _log_int(rng, 1, 250)
        most = 300 if kind == "plugin" else 2000
        return {"kind": kind, "reads": _log_int(rng, 3, most), "haps": rng.randint(1, 64), "read_lo": lo, "read_hi": hi,
                "hap_len": hi + _log_int(rng, 10, 400)}
    lo, hi = {"batch": (20, 1000), "compute": (10, 6000), "stream": (20, 400), "long": (2, 16), "double": (3, 100),
              "calib": (40, 700), "pd": (10, 600), "raw": (10, 400), "realign": (20, 1000)}[kind]
    case = {"kind": kind, "regions": _log_int(rng, lo, hi)}
    if kind == "raw":
        case["imputation"] = rng.choice(["dragstr", "pcr"])
    return case


# ------------------------------------------------------------------------------------------------ inputs
def _one_region(case, rng):
    """One region: haplotypes that are variants of one random sequence, reads sampled from them at random offsets
    (1 % substitutions, 0.1 % indels), base qualities uniform in 10..40, gap open 45, continuation 10."""
    acgt = np.frombuffer(b"ACGT", dtype=np.uint8)
    base = acgt[rng.integers(0, 4, case["hap_len"])]
    haps = [base]
    for _ in range(1, case["haps"]):
        h = base.copy()
        for _ in range(int(rng.integers(1, 4))):
            p = int(rng.integers(0, len(h) - 12))
            what = int(rng.integers(0, 3))
            n = int(rng.integers(1, 11))
            if what == 0:
                h[p] = acgt[rng.integers(0, 4)]
            elif what == 1:
                h = np.concatenate([h[:p], acgt[rng.integers(0, 4, n)], h[p:]])
            elif len(h) - n > case["read_hi"]:
                h = np.concatenate([h[:p], h[p + n:]])
        haps.append(h)
    reads = []
    for _ in range(case["reads"]):
        n = int(rng.integers(case["read_lo"], case["read_hi"] + 1))
        h = haps[int(rng.integers(0, len(haps)))]
        o = int(rng.integers(0, len(h) - n + 1))
        b = h[o:o + n].copy()
        sub = rng.random(n) < 0.01
        b[sub] = acgt[rng.integers(0, 4, int(sub.sum()))]
        if rng.random() < 0.001 * n:
            p = int(rng.integers(1, n))
            b = np.concatenate([b[:p], acgt[rng.integers(0, 4, 1)], b[p:-1]])
        reads.append((b, rng.integers(10, 41, n).astype(np.uint8), np.full(n, 45, np.uint8), np.full(n, 45, np.uint8),
                      np.full(n, 10, np.uint8)))
    return haps, reads


def _inputs(case, seed):
    """The case's reads and haplotypes in host memory.  The generated regions' sizes are those of the generator's own
    seed; the seed here draws the sequences (the four letters permuted per region) and every base quality anew."""
    if case["kind"] in ("plugin", "region"):
        return _one_region(case, np.random.default_rng([seed, case["reads"], case["haps"], case["hap_len"]]))
    which = {"long": 2, "calib": 3, "stream": 4}.get(case["kind"], 1)
    wl = workload.generate(which, regions=case["regions"])
    rng = np.random.default_rng([seed, case["regions"]])
    letters = np.zeros((wl.n_regions, 256), dtype=np.uint8)
    letters[:, list(b"ACGT")] = rng.permuted(np.tile(np.frombuffer(b"ACGT", np.uint8), (wl.n_regions, 1)), axis=1)
    low, high = (5, 25) if which == 2 else (10, 40)
    wl.quals[:] = rng.integers(low, high + 1, len(wl.quals), dtype=np.uint8)
    for g in range(wl.n_regions):
        for flat, off, inner in ((wl.bases, wl.read_off, wl.region_read_off), (wl.hap_bases, wl.hap_off, wl.region_hap_off)):
            part = flat[off[inner[g]]:off[inner[g + 1]]]
            part[:] = letters[g][part]
    return wl


def _mapq(wl, seed):
    return np.random.default_rng([seed, 7]).integers(20, 61, wl.n_reads).astype(np.int32)


def _dragstr_tables():
    """Gap open / continuation tables [8 periods][20 repeats]: open falls with the repeat count, continuation by period."""
    p, r = np.arange(1, 9)[:, None], np.arange(1, 21)[None, :]
    gop = np.clip(45.0 - 1.4 * (r - 1) - 0.6 * (p - 1), 12.0, 45.0)
    return gop, np.repeat(np.round(1000.0 / p) / 100.0, 20, axis=1)


def _engine(double=False):
    if double not in _ENGINES:
        _ENGINES[double] = Engine(use_double_precision=double)
    return _ENGINES[double]


class _State(dict):
    """A state whose held batch is given back with it."""

    def __del__(self):
        if "batch" in self:
            self["batch"].close()


def prepare(case, seed):
    kind = case["kind"]
    data = _inputs(case, seed)
    s = _State(kind=kind)
    if kind == "plugin":
        if "plugin" not in _ENGINES:
            _ENGINES["plugin"] = CudaLoglessPairHMM(PairHMMNativeArguments())
        s["haps"], s["reads"] = data
        return s
    if kind == "region":
        data = workload.from_pairs([data])
    s["wl"], s["engine"] = data, _engine(kind == "double")
    if kind in ("batch", "realign"):
        s["batch"] = s["engine"].batch(data)
        if kind == "realign":
            s["batch"].forward()
            s["batch"].results()
    elif kind == "stream":
        if "queue" not in _ENGINES:
            _ENGINES["queue"] = s["engine"].queue()
    elif kind == "calib":
        s["set"] = calibration.CalibrationSet(data)
        g = torch.Generator().manual_seed(seed)
        s["theta"] = (calibration.default_theta() - 0.3 * torch.rand(8, 20, 2, generator=g)).cuda()
    elif kind == "pd":
        s["flags"] = workload.pd_flags(data, seed)
    elif kind == "raw":
        s["mapq"] = _mapq(data, seed)
        s["dragstr"] = _dragstr_tables() if case["imputation"] == "dragstr" else None
    return s


def _alignments(best, informative, aln):
    ops = np.zeros(8 * len(best) + 64, dtype=np.uint32)  # as many values whatever the number of cigar elements
    ops[:len(aln.cigar_ops)] = aln.cigar_ops
    return {"best": best, "informative": informative, "offset": aln.offset, "cigar_len": aln.cigar_len, "cigar_ops": ops}


def run(s):
    kind = s["kind"]
    if kind == "plugin":
        hmm = _ENGINES["plugin"]
        hmm.initialize(s["haps"])
        return hmm.compute_log10_likelihoods(s["reads"])
    eng, wl = s["engine"], s["wl"]
    if kind in ("region", "compute", "long", "double"):
        return eng.compute(wl)
    if kind == "batch":
        s["batch"].forward()
        return s["batch"].results()
    if kind == "stream":
        q = _ENGINES["queue"]
        out = q.push(wl)
        q.flush()
        return out
    if kind == "calib":
        theta = s["theta"].detach().clone().requires_grad_(True)
        ll = calibration.log10_likelihoods(theta, s["set"], eng)
        ll.sum().backward()
        return {"log10": ll.detach(), "grad": theta.grad}
    if kind == "pd":
        return eng.pd_compute(wl, s["flags"])
    if kind == "realign":
        return _alignments(*smithwaterman.realign_batch(s["batch"]))
    with eng.raw_batch(wl, s["mapq"], dragstr=s["dragstr"]) as b:
        b.forward()
        keep = b.postprocess()
        out = b.results()
        return {"log10": out, "keep": keep, **_alignments(*smithwaterman.realign_batch(b))}


def work(case):
    """Reads and haplotypes in (5 bytes a read base, 1 a haplotype base), results out; 11 FLOP a cell of the forward
    (M: add, mul, fma, mul; I and D: fma), 12 integer operations a cell of the alignment, 33 for forward + backward."""
    kind = case["kind"]
    if kind in ("plugin", "region"):
        rb = case["reads"] * (case["read_lo"] + case["read_hi"]) / 2
        hb = case["haps"] * case["hap_len"]
        return {"bytes": 5.0 * rb + hb + 8.0 * case["reads"] * case["haps"], "flops": 11.0 * rb * hb}
    g = case["regions"]
    if kind == "calib":  # 8 reads of 150 bases x 1 haplotype of 300
        return {"bytes": g * (8 * 150 * (2 + 8 + 8) + 300 + 8 * 8.0), "flops": 33.0 * g * 8 * 150 * 300}
    if kind == "long":   # 36 reads of 1,400 bases x 10 haplotypes of 2,250
        return {"bytes": g * (36 * 1400 * 5 + 10 * 2250 + 36 * 10 * 8.0), "flops": 11.0 * g * 36 * 1400 * 10 * 2250}
    reads, haps = MEAN_READS, MEAN_HAPS
    rb, hb, pairs = reads * MEAN_READ_LEN, haps * MEAN_HAP_LEN, reads * haps
    if kind == "stream":  # 5 % of the regions: 2,000 reads x 64 haplotypes
        cells = 0.95 * rb * hb + 0.05 * 2000 * MEAN_READ_LEN * 64 * MEAN_HAP_LEN
        rb, hb = 0.95 * rb + 0.05 * 2000 * MEAN_READ_LEN, 0.95 * hb + 0.05 * 64 * MEAN_HAP_LEN
        pairs = 0.95 * pairs + 0.05 * 2000 * 64
        return {"bytes": g * (5 * rb + hb + 8 * pairs), "flops": 11.0 * g * cells}
    if kind == "realign":  # each read once against its best haplotype; likelihoods in, cigars out
        return {"bytes": g * (rb + hb + 8 * pairs + 24 * reads), "flops": 12.0 * g * rb * MEAN_HAP_LEN * 0.84}
    extra = 12.0 * rb * MEAN_HAP_LEN * 0.84 if kind == "raw" else 0.0
    return {"bytes": g * (5 * rb + hb * (2 if kind == "pd" else 1) + 8 * pairs), "flops": g * (11.0 * rb * hb + extra)}


# ------------------------------------------------------------------------------------------------ 64-bit values
def _phred_tables(dev):
    """Error probability per Phred value and matchToMatch per (insertion, deletion) pair, as PairHMMModel defines
    them: log10(10^-i/10 + 10^-d/10) through the Jacobian table of step 1e-4 up to 8, then 1 - 10^that."""
    q = np.arange(256, dtype=np.float64)
    err = 10.0 ** (np.minimum(q, 254) / -10.0)
    cache = np.log10(1.0 + 10.0 ** (-np.arange(80001) * 0.0001))
    i, j = np.meshgrid(np.arange(128), np.arange(128), indexing="ij")
    lo, hi = -0.1 * np.maximum(i, j), -0.1 * np.minimum(i, j)
    diff = hi - lo
    add = np.where(diff < 8.0, cache[np.minimum((diff * (1.0 / 0.0001) + 0.5).astype(np.int64), 80000)], 0.0)
    total = 10.0 ** (hi + add)
    mm = np.where(total >= 1.0, 0.0, 10.0 ** (np.log1p(-np.where(total >= 1.0, 0.0, total)) / math.log(10.0)))
    return torch.from_numpy(err).to(dev), torch.from_numpy(mm).to(dev)


def _spans(flat, off, idx, width, fill, lead=0, tail=0):
    """Rows flat[off[k] : off[k + 1]] for k in idx as one matrix, `lead` columns of fill before and padding behind."""
    a, n = off[idx], off[idx + 1] - off[idx]
    c = torch.arange(-lead, width + tail, device=flat.device)
    inside = (c[None, :] >= 0) & (c[None, :] < n[:, None])
    at = (a[:, None] + c[None, :]).clamp_(0, flat.numel() - 1)
    return torch.where(inside, flat[at], torch.as_tensor(fill, dtype=flat.dtype, device=flat.device))


def _forward64(wl, planes, flags=None):
    """log10 likelihood of every pair (LoglessPairHMM, or LoglessPDPairHMM with flags), swept by anti-diagonals."""
    dev = torch.device("cuda")
    err, m2m = _phred_tables(dev)
    prob = 1.0 - err
    up = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev)  # noqa: E731
    bases, quals, ins, dels, gcp = (up(x) for x in planes)
    read_off, hap_off, hap = up(wl.read_off), up(wl.hap_off), up(wl.hap_bases)
    pd = up(flags) if flags is not None else None
    pr, ph = (up(x) for x in wl.pair_index())
    R, H = read_off[pr + 1] - read_off[pr], hap_off[ph + 1] - hap_off[ph]
    order = torch.argsort((R // 16) * 65536 + H)
    out = torch.empty(wl.n_pairs, dtype=torch.float64, device=dev)
    k = 0
    while k < len(order):
        idx = order[k:k + max(1, 24_000_000 // max(1, int(R[order[k]]) + 16))]
        k += len(idx)
        out[idx] = _sweep64(idx, pr, ph, R, H, bases, quals, ins, dels, gcp, read_off, hap, hap_off, pd, err, prob, m2m)
    return out.cpu().numpy()


def _column_states(pd):
    """Per column NORMAL 0, INSIDE_DEL 1, AFTER_DEL 2: the state the flags of the columns before it set."""
    st = torch.zeros_like(pd)
    cur = torch.zeros_like(pd[:, 0])
    for c in range(pd.shape[1]):
        st[:, c] = cur
        cur = torch.where(cur == 2, 0, cur)
        cur = torch.where((pd[:, c] & 2) != 0, 1, cur)
        cur = torch.where((pd[:, c] & 4) != 0, 2, cur)
    return st


def _sweep64(idx, pr, ph, R, H, bases, quals, ins, dels, gcp, read_off, hap, hap_off, pd, err, prob, m2m):
    r, h, R, H = pr[idx], ph[idx], R[idx], H[idx]
    Rm, Hm = int(R.max()), int(H.max())
    row = lambda x, fill: _spans(x, read_off, r, Rm, fill)  # noqa: E731
    x, q, i_, d_, g = row(bases, 0), row(quals, 0).long(), row(ins, 40).long(), row(dels, 40).long(), row(gcp, 10).long()
    pm, pe = prob[q], err[q] / 3.0
    mm, im, mi, ii, md = m2m[i_, d_], prob[g], err[i_], err[g], err[d_]
    flip = lambda y: _spans(y, hap_off, h, Hm, 0, lead=Rm, tail=Rm).flip(1)  # noqa: E731
    F = flip(hap)
    x_n = x == 78
    if pd is not None:
        states = _column_states(_spans(pd, hap_off, h, Hm, 0))
        FS = torch.nn.functional.pad(states, (Rm, Rm)).flip(1)
        FP = flip(pd)
        bit = torch.zeros_like(x)
        for c, b in ((65, 8), (67, 16), (71, 32), (84, 64)):
            bit = torch.where(x == c, b, bit)
    n = len(idx)
    zeros = lambda: torch.zeros(n, Rm + 1, dtype=torch.float64, device=x.device)  # noqa: E731
    init = (2.0 ** 1020 / H.double())
    sets = []
    for _ in range(3):  # M, I, D (and the branch states) of three anti-diagonals
        t = [zeros() for _ in range(3 if pd is None else 6)]
        t[2][:, 0] = init
        sets.append(t)
    acc = torch.zeros(n, dtype=torch.float64, device=x.device)
    lane = torch.arange(n, device=x.device)
    p2, p1, cur = sets
    r_lo = int(R.min())
    for d in range(2, Rm + Hm + 1):
        w = Rm + Hm - d + 1
        y = F[:, w:w + Rm]
        m = (x == y) | x_n | (y == 78)
        if pd is not None:
            f, st = FP[:, w:w + Rm], FS[:, w:w + Rm]
            m |= ((f & 1) != 0) & ((f & bit) != 0)
        prior = torch.where(m, pm, pe).mul_(y != 0)
        M2, I2, D2, M1, I1, D1 = p2[0], p2[1], p2[2], p1[0], p1[1], p1[2]
        a, b, c, left_m, left_d, up_m, up_i = (M2[:, :-1], I2[:, :-1], D2[:, :-1], M1[:, 1:], D1[:, 1:], M1[:, :-1],
                                               I1[:, :-1])
        if pd is not None:
            after, inside, end = st == 2, st == 1, (f & 4) != 0
            for k, v in enumerate((M1, I1, D1)):
                old = p1[3 + k][:, 1:]
                here = torch.where(after, torch.maximum(old, v[:, 1:]), torch.where(inside, old, v[:, 1:]))
                cur[3 + k][:, 1:] = here.mul_(y != 0)
            pick = lambda on, p, q_: torch.where(on, torch.maximum(p, q_), q_)  # noqa: E731
            a, b, c = (pick(after, p2[3 + k][:, :-1], v) for k, v in enumerate((a, b, c)))
            left_m, left_d = pick(after, p1[3][:, 1:], left_m), pick(after, p1[5][:, 1:], left_d)
            up_m, up_i = pick(end, p1[3][:, :-1], up_m), pick(end, p1[4][:, :-1], up_i)
        new_m = (b + c).mul_(im).addcmul_(a, mm).mul_(prior)
        new_i = (up_m * mi).addcmul_(up_i, ii)
        new_d = (left_m * md).addcmul_(left_d, ii)
        cur[0][:, 1:], cur[1][:, 1:], cur[2][:, 1:] = new_m, new_i, new_d
        if d > r_lo:
            last = cur[0][lane, R] + cur[1][lane, R]
            acc += torch.where((d - R >= 1) & (d - R <= H), last, 0.0)
        p2, p1, cur = p1, cur, p2
    return torch.log10(acc) - 1020.0 * math.log10(2.0)


def _dragstr64(wl, quals, mapq):
    """The read planes after the mapping-quality cap, the base-quality threshold (18, floor 6) and the DRAGstr
    imputation: per position the repeat count of the most repeated period (ties to the shorter one), looked up in
    the tables; 45 / 10 at the last base."""
    gop_t, gcp_t = _dragstr_tables()
    off, n = wl.read_off, np.diff(wl.read_off)
    q = np.minimum(quals, np.repeat(mapq, n).astype(np.uint8))
    q = np.where(q < 18, 6, q).astype(np.uint8)
    width = int(n.max()) + 9
    cols = np.arange(width)
    inside = cols[None, :] < n[:, None]
    b = np.where(inside, wl.bases[np.minimum(off[:-1, None] + cols, len(wl.bases) - 1)].astype(np.int16), -1 - (cols % 16))
    best, period = np.zeros(b.shape, np.int64), np.ones(b.shape, np.int64)
    for p in range(1, 9):
        same = np.zeros(b.shape, bool)
        same[:, :-p] = (b[:, :-p] == b[:, p:]) & inside[:, p:]
        fwd, bwd = np.zeros(b.shape, np.int64), np.zeros(b.shape, np.int64)
        for c in range(width - 2, -1, -1):
            fwd[:, c] = np.where(same[:, c], fwd[:, c + 1] + 1, 0)
        for c in range(1, width):
            bwd[:, c] = np.where(same[:, c - 1], bwd[:, c - 1] + 1, 0)
        unit = np.where(cols[None, :] + p <= n[:, None], 1 + fwd // p + bwd // p, 0)
        count = np.zeros(b.shape, np.int64)
        for k in range(-(p - 1), 2):  # unit starts in pos - p + 1 .. pos + 1
            src = np.clip(cols + k, 0, width - 1)
            v = np.where((cols + k >= 0) & (cols + k < width), unit[:, src], 0)
            short = (cols + k == 0) & (cols < p - 1)
            count = np.maximum(count, np.where(short[None, :] & (v > 0), np.maximum(1, v - 1), v))
        more = count > best
        best, period = np.where(more, count, best), np.where(more, p, period)
    at = (period - 1, np.clip(best, 1, 20) - 1)
    gop = np.floor(np.minimum(40.0, gop_t[at]) + 0.5)
    gcp = np.floor(gcp_t[at] + 0.5)
    last = cols[None, :] == n[:, None] - 1
    gop, gcp = np.where(last, 45, gop)[inside].astype(np.uint8), np.where(last, 10, gcp)[inside].astype(np.uint8)
    return wl.bases, q, gop, gop, gcp


def _calibration64(case, seed):
    """log10 L of each pair with MI = MD = 10^g, MM = 1 - 2 10^g, II = DD = 10^c, IM = 1 - 10^c per read position,
    and the gradient of their sum in the table, by torch's autograd in 64 bits."""
    s = prepare(case, seed)
    wl, dev = s["wl"], torch.device("cuda")
    theta = s["theta"].double().requires_grad_(True)
    index = torch.from_numpy(s["set"].param_index_np).to(dev)
    flat = theta.reshape(-1, 2)[index.clamp(min=0)]
    fixed = (index < 0)[:, None]
    gc = torch.where(fixed, torch.tensor([-4.5, -1.0], dtype=torch.float64, device=dev), flat)
    up = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev)  # noqa: E731
    pr, ph = (up(x) for x in wl.pair_index())
    R, H = int(wl.read_lengths()[0]), int(wl.hap_lengths()[0])  # every read 150 bases, every haplotype 300
    g, c = gc[:, 0].reshape(-1, R)[pr], gc[:, 1].reshape(-1, R)[pr]
    x, q = up(wl.bases).reshape(-1, R)[pr], up(wl.quals).reshape(-1, R)[pr].long()
    err, _ = _phred_tables(dev)
    pm, pe = 1.0 - err[q], err[q] / 3.0
    hb = up(wl.hap_bases).reshape(-1, H)[ph]
    F = torch.nn.functional.pad(hb, (R, R)).flip(1)
    mi, ii = 10.0 ** g, 10.0 ** c
    mm, im = 1.0 - 2.0 * mi, 1.0 - ii
    n = len(pr)
    zero = torch.zeros(n, R, dtype=torch.float64, device=dev)
    top = torch.zeros(n, 1, dtype=torch.float64, device=dev)
    init = top + 1.0 / H
    M1 = I1 = D1 = M2 = I2 = D2 = zero
    down = lambda v, t: torch.cat([t, v[:, :-1]], 1)  # noqa: E731
    acc = torch.zeros(n, dtype=torch.float64, device=dev)
    for d in range(2, R + H + 1):
        w = R + H - d + 1
        y = F[:, w:w + R]
        prior = torch.where(x == y, pm, pe) * (y != 0)
        M = prior * (down(M2, top) * mm + (down(I2, top) + down(D2, init)) * im)
        I = down(M1, top) * mi + down(I1, top) * ii
        D = M1 * mi + D1 * ii
        if d > R:
            acc = acc + M[:, -1] + I[:, -1]
        M2, I2, D2, M1, I1, D1 = M1, I1, D1, M, I, D
    ll = torch.log10(acc)
    ll.sum().backward()
    return {"log10": ll.detach(), "grad": theta.grad}


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind in ("plugin", "region"):
            wl = workload.from_pairs([_inputs(case, seed)])
            return _forward64(wl, (wl.bases, wl.quals, wl.ins, wl.dels, wl.gcp))
        if kind == "realign":
            return None  # whole numbers
        if kind == "raw" and case["imputation"] != "dragstr":
            return None  # the repeat search of the PCR model, position by position, takes too long here
        if kind != "calib":
            wl = _inputs(case, seed)
            if wl.cells() > 1.6e11:
                return None  # over 20 seconds
            if kind == "pd":
                return _forward64(wl, (wl.bases, wl.quals, wl.ins, wl.dels, wl.gcp), workload.pd_flags(wl, seed))
            if kind != "raw":
                return _forward64(wl, (wl.bases, wl.quals, wl.ins, wl.dels, wl.gcp))
            out = _forward64(wl, _dragstr64(wl, wl.quals, _mapq(wl, seed)))
            nh = np.diff(wl.region_hap_off)
            for g in range(wl.n_regions):  # normalisation: no likelihood more than 4.5 below the read's best
                block = out[wl.out_off[g]:wl.out_off[g + 1]].reshape(-1, nh[g])
                np.maximum(block, block.max(axis=1, keepdims=True) - 4.5, out=block)
            return {"log10": out, "keep": None, "best": None, "informative": None, "offset": None, "cigar_len": None,
                    "cigar_ops": None}
    return _calibration64(case, seed)
