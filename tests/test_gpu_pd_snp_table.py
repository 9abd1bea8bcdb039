"""Undetermined SNP columns through the packed PD kernel's prior table: at every distance around the one from which on a
column may take the table (63 behind the last), across haplotype boundaries, with one and two alternatives, in one and
several strips, with deletions beside them."""
import numpy as np
import pytest

from gatk_gb300 import native, workload
from gatk_gb300.pairhmm import Engine
from oracle import oracle

pytestmark = pytest.mark.gpu

BIT = {65: 8, 67: 16, 71: 32, 84: 64}


def _region(rng, read_lengths, hap_len, gap, alternatives, deletion):
    acgt = np.frombuffer(b"ACGT", np.uint8)
    haps, flags = [], []
    for first in (0, 1, 30, hap_len - 63, hap_len - 2):
        h, f = acgt[rng.integers(0, 4, hap_len)], np.zeros(hap_len, np.uint8)
        for j in range(max(first, 0), hap_len, gap):
            others = [c for c in acgt if c != h[j]]
            f[j] |= 1
            for k in range(alternatives):
                f[j] |= BIT[int(others[(j + k) % 3])]
        if deletion:
            a = hap_len // 2
            f[a] |= 2
            f[a + 3] |= 4
        haps.append(h)
        flags.append(f)
    reads = []
    for n in read_lengths:
        h = haps[int(rng.integers(0, len(haps)))]
        o = int(rng.integers(0, max(1, len(h) - n + 1)))
        b = np.resize(h[o:], n).copy()
        miss = rng.random(n) < 0.02
        b[miss] = acgt[rng.integers(0, 4, int(miss.sum()))]
        reads.append((b, rng.integers(10, 41, n), np.full(n, 45), np.full(n, 45), np.full(n, 10)))
    return haps, flags, reads


@pytest.mark.parametrize("gap,alternatives,deletion", [(1, 1, False), (31, 2, False), (62, 1, True), (63, 1, True),
                                                       (63, 2, False), (64, 2, True), (130, 1, True)])
def test_snp_columns(gap, alternatives, deletion):
    rng = np.random.default_rng([gap, alternatives])
    haps, flags, reads = _region(rng, [20, 62, 95, 126, 150, 190, 222, 250, 300], 170, gap, alternatives, deletion)
    eng = Engine()
    try:
        copies = 640  # enough work for whole regions a task, so that haplotypes follow one another in a stream
        wl = workload.from_pairs([(haps, reads)] * copies)
        with eng.pd_batch(wl, np.concatenate(flags * copies)) as b:
            b.forward(native.MODE_PD_FP32)
            together = b.results().reshape(copies, len(reads), len(haps))
        alone = np.stack([eng.pd_compute(workload.from_pairs([([h], reads)]), f) for h, f in zip(haps, flags)], axis=1)
    finally:
        eng.close()
    assert np.array_equal(together, np.broadcast_to(alone, together.shape))
    one = workload.from_pairs([(haps, reads)])
    want = oracle.pd_compute_workload(one, np.concatenate(flags)).reshape(alone.shape)
    assert np.abs(alone - want).max() <= 1e-3  # the bar of FP32 results
