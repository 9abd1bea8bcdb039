"""Haplotypes of fewer than 63 columns among longer ones in one FP32 task: the same bits as each haplotype in a task of its
own, wherever the short ones stand, and little time for the others."""
import numpy as np
import pytest

from gatk_gb300 import native, workload
from gatk_gb300.pairhmm import Engine
from oracle import oracle

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _region(rng, read_lengths, hap_lengths):
    """Related haplotypes, leading parts of one sequence, and reads of them, so that most pairs keep FP32 results."""
    seq = ACGT[rng.integers(0, 4, max(hap_lengths))]
    reads = []
    for n in read_lengths:
        o = int(rng.integers(0, max(1, min(200, len(seq) - n))))
        b = np.resize(seq[o:o + n], n)
        reads.append((b, rng.integers(20, 41, n), np.full(n, 45), np.full(n, 45), np.full(n, 10)))
    return [seq[:n] for n in hap_lengths], reads


@pytest.mark.parametrize("haps", [
    (62, 200), (200, 62), (1, 1, 1, 200), (200, 1, 1, 1), (63, 62, 63, 62, 64), (62, 62, 62, 62), (200, 62, 126, 300),
    (300, 5, 63, 5, 63, 200), (40, 200, 210, 1, 220, 2, 3, 230, 62), (63, 63, 63)], ids=str)
def test_bits_are_those_of_one_haplotype_a_task(haps):
    rng = np.random.default_rng(21)
    region = _region(rng, [2, 30, 31, 62, 94, 126, 127, 190, 254, 255, 300, 520, 521] + list(range(40, 140, 3)), haps)
    one = workload.from_pairs([region])
    eng = Engine()
    try:
        eng.set_tuning(chunk_cols=1)  # a haplotype a task
        with eng.batch(one) as b:
            b.forward(native.MODE_FP32_RERUN)
            alone = b.results()
        eng.set_tuning()
        copies = 400  # enough work for whole regions a task
        with eng.batch(workload.from_pairs([region] * copies)) as b:
            b.forward(native.MODE_FP32_RERUN)
            together = b.results().reshape(copies, -1)
    finally:
        eng.close()
    assert np.array_equal(together, np.broadcast_to(alone, together.shape))
    assert np.abs(alone - oracle.compute_workload(one)).max() <= 1e-3


def test_one_short_haplotype_costs_little():
    """24 haplotypes of 400 columns and one of 62 in a task: 125 of its 9,700 steps are checked against the column codes,
    each less than three plain steps' time, 3 % of the task; with every step checked it is half as long again.  1.15
    leaves the rest for noise."""
    rng = np.random.default_rng(22)
    ms = {}
    eng = Engine()
    try:
        for short in (63, 62):
            region = _region(rng, [150, 151, 200, 250] * 16, [400] * 12 + [short] + [400] * 12)
            with eng.batch(workload.from_pairs([region] * 500)) as b:
                times = []
                for _ in range(6):
                    b.forward(native.MODE_FP32_RERUN)
                    times.append(b.stats()["ms_fp32"])
                ms[short] = min(times)
    finally:
        eng.close()
    assert ms[62] <= 1.15 * ms[63], ms


@pytest.mark.parametrize("copies", [3, 900])
def test_mixed_and_long_regions_in_one_batch(copies):
    """Few of both go to one kernel, many to one each."""
    rng = np.random.default_rng(23)
    reads = [94, 126, 190, 200, 254, 255, 300, 520] + list(range(60, 140, 5))
    regions = [_region(rng, reads, haps) for haps in ((300, 62, 200, 400), (300, 310, 63), (50, 55, 70, 62))]
    eng = Engine()
    try:
        alone = [eng.compute(workload.from_pairs([r])) for r in regions]
        with eng.batch(workload.from_pairs(regions * copies)) as b:
            b.forward(native.MODE_FP32_RERUN)
            together = b.results().reshape(copies, -1)
    finally:
        eng.close()
    want = np.concatenate(alone)
    assert np.array_equal(together, np.broadcast_to(want, together.shape))
    assert np.abs(want - oracle.compute_workload(workload.from_pairs(regions))).max() <= 1e-3
