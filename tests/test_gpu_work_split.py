"""How a call's work is split must not show in its results: FP64 pairs on one warp or one block, strips of any height,
and regions cut into more or fewer FP32 tasks."""
import numpy as np
import pytest

from gatk_gb300 import native, workload
from gatk_gb300.pairhmm import Engine
from oracle import oracle

pytestmark = pytest.mark.gpu


def _reads(rng, lengths, ins=(30, 46)):
    acgt = np.frombuffer(b"ACGT", np.uint8)
    return [(acgt[rng.integers(0, 4, n)], rng.integers(6, 41, n), rng.integers(*ins, n), rng.integers(*ins, n),
             np.full(n, 10)) for n in lengths]


def _region(rng, read_lengths, hap_lengths, ins=(30, 46)):
    acgt = np.frombuffer(b"ACGT", np.uint8)
    return [acgt[rng.integers(0, 4, n)] for n in hap_lengths], _reads(rng, read_lengths, ins)


EDGES = [1, 2, 31, 32, 33, 64, 65, 96, 97, 128, 129, 160, 161, 192, 224, 255, 256, 257, 289, 384, 385]


@pytest.mark.parametrize("case", ["pair_per_block", "pair_per_warp", "long_reads", "exact_tier"])
def test_fp64_strip_shapes(case):
    """Reads at the edges of the strips' heights, haplotypes at the edges of the 16-column phases.  |d| <= 1e-9 is the
    repository's bar for FP64 results."""
    rng = np.random.default_rng(11)
    haps = [1, 2, 15, 16, 17, 31, 32, 33, 48, 97]
    if case == "pair_per_block":
        regions = [_region(rng, EDGES, haps)]
    elif case == "pair_per_warp":  # more pairs than any grid has warps, no read of 481 bases or more
        regions = [_region(rng, EDGES, haps) for _ in range(16)]
    elif case == "long_reads":
        regions = [_region(rng, [480, 481, 512, 513, 640, 1025, 1537, 2049], [1, 16, 130, 700])]
    else:  # insertion and deletion penalties of Phred 3: matchToMatch about 0, every pair in the unscaled tier
        regions = [_region(rng, EDGES, haps, ins=(3, 4))]
    wl = workload.from_pairs(regions)
    eng = Engine(use_double_precision=True)
    try:
        got = eng.compute(wl)
    finally:
        eng.close()
    want = oracle.compute_workload(wl)
    differ = got != want  # (infinities are equal)
    assert np.max(np.abs(got[differ] - want[differ]), initial=0.0) <= 1e-9


def test_fp64_runs_of_haplotypes():
    """Enough pairs for a warp to take runs of a read's haplotypes as one stream: short, empty and ordinary haplotypes
    following one another, results ending several to a phase of 16 columns.  |d| <= 1e-9 as above."""
    rng = np.random.default_rng(15)
    haps = [1, 2, 15, 16, 17, 0, 31, 32, 33, 3, 3, 3, 3, 48, 97, 210, 0, 0, 130]
    wl = workload.from_pairs([_region(rng, EDGES, haps) for _ in range(60)])  # 23,940 pairs
    eng = Engine(use_double_precision=True)
    try:
        got = eng.compute(wl)
    finally:
        eng.close()
    want = oracle.compute_workload(wl)
    differ = got != want  # (infinities are equal)
    assert np.max(np.abs(got[differ] - want[differ]), initial=0.0) <= 1e-9


def test_results_do_not_depend_on_the_task_split():
    """Regions called one by one (cut down to a haplotype a task) and in one batch of many (whole regions a task) give
    the same bits, several strips included."""
    rng = np.random.default_rng(12)
    few = [_region(rng, [40, 150, 151, 254, 255, 300, 520], [700, 640, 655, 610, 620]),
           _region(rng, [1, 30, 31, 62, 63], [90]), _region(rng, [100, 101, 102], [333] * 9)]
    eng = Engine()
    try:
        alone = [eng.compute(workload.from_pairs([r])) for r in few]
        big = workload.generate(1, regions=400)
        haps_reads = [([big.hap(h) for h in range(int(big.region_hap_off[g]), int(big.region_hap_off[g + 1]))],
                       [big.read(r) for r in range(int(big.region_read_off[g]), int(big.region_read_off[g + 1]))])
                      for g in range(0, 400, 4)]
        wl = workload.from_pairs(few + haps_reads * 4)
        with eng.batch(wl) as b:
            b.forward(native.MODE_FP32_RERUN)
            together = b.results()
    finally:
        eng.close()
    assert np.array_equal(np.concatenate(alone), together[:sum(len(a) for a in alone)])


def test_short_haplotype_in_a_task_changes_no_other_result():
    """A haplotype of fewer than 63 columns sends its task's steps through the checked form; the other haplotypes' results
    keep every bit, at the lengths around that limit, in one and several strips."""
    rng = np.random.default_rng(13)
    region = _region(rng, [2, 30, 31, 62, 94, 126, 158, 190, 222, 254, 300, 520, 521] + list(range(60, 200, 3)),
                     [63, 64, 65, 126, 127, 200, 90])
    short = _region(rng, [1], [62, 1, 40])[0]
    haps, reads = region
    out = {}
    eng = Engine()
    try:
        for name, hs in (("long", haps), ("mixed", [short[0]] + haps[:3] + [short[1]] + haps[3:] + [short[2]])):
            with eng.batch(workload.from_pairs([(hs, reads)] * 256)) as b:  # enough work for whole regions a task
                b.forward(native.MODE_FP32_RERUN)
                out[name] = b.results().reshape(256, len(reads), len(hs))
    finally:
        eng.close()
    assert np.array_equal(out["mixed"][:, :, [1, 2, 3, 5, 6, 7, 8]], out["long"])
    want = oracle.compute_workload(workload.from_pairs([(haps, reads)])).reshape(len(reads), len(haps))
    assert np.abs(out["long"] - want).max() <= 1e-3



RING_HAPS = (287, 288, 289, 319, 320, 321, 352, 543, 544, 545)


@pytest.mark.parametrize("related", [False, True])
def test_strip_boundaries_around_the_ring(related):
    """Reads of several strips against haplotypes whose lengths sit around the 32 columns in which a strip's boundary row
    is read back: one haplotype a task and several, the same bits, and the oracle's values within the FP32 bar.  Unrelated
    haplotypes: each read fits one, the other pairs go on to FP64; related: leading parts of one sequence, so that most
    pairs keep their FP32 results."""
    rng = np.random.default_rng(14)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    haps = [acgt[rng.integers(0, 4, n)] for n in RING_HAPS]
    if related:
        haps = [haps[-1][:n] for n in RING_HAPS]
    reads = []
    for n in (255, 256, 270, 286, 509, 510, 511, 540):
        for h in [x for x in haps if len(x) >= n][:3]:
            o = int(rng.integers(0, len(h) - n + 1))
            reads.append((h[o:o + n], rng.integers(30, 41, n), np.full(n, 45), np.full(n, 45), np.full(n, 10)))
    one = workload.from_pairs([(haps, reads)])
    eng = Engine()
    try:
        alone = eng.compute(one)
        copies = 128
        with eng.batch(workload.from_pairs([(haps, reads)] * copies)) as b:
            b.forward(native.MODE_FP32_RERUN)
            together = b.results().reshape(copies, -1)
    finally:
        eng.close()
    assert np.array_equal(together, np.broadcast_to(alone, together.shape))
    assert np.abs(alone - oracle.compute_workload(one)).max() <= 1e-3
