"""The FP32 strip scratch of a batch: each bucket's part for its own longest task, 16 bytes a column and warp; and batches
of other part sizes through the same buffers, one after the other."""
import numpy as np
import pytest

from gatk_gb300 import native, workload
from gatk_gb300.pairhmm import Engine

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _region(rng, n_reads, read_length, hap_length):
    hap = ACGT[rng.integers(0, 4, hap_length)]
    reads = []
    for _ in range(n_reads):
        o = int(rng.integers(0, hap_length - read_length + 1))
        n = read_length
        reads.append((hap[o:o + n], rng.integers(20, 41, n), np.full(n, 45), np.full(n, 45), np.full(n, 10)))
    return [hap], reads


def _kept_bytes(regions):
    eng = Engine()
    try:
        with eng.batch(workload.from_pairs(regions)) as b:
            b.forward(native.MODE_FP32_RERUN)
        return eng.trim()
    finally:
        eng.close()


def test_size():
    """Four tasks of 10,000 columns in one bucket, 400 of 600 in another: 4 x 10,000 x 16 + 400 x 600 x 16 bytes, 4.5 MB;
    sized by blocks of four warps and the longest column count of all, 97 to 65 MB.  The other buffers of the two batches
    differ by the longer reads' bytes, 0.5 MB (five planes, pinned and device)."""
    rng = np.random.default_rng(31)
    long_hap = _region(rng, 8, 300, 10000)
    strips = _kept_bytes([long_hap, _region(rng, 800, 520, 600)])
    single = _kept_bytes([long_hap, _region(rng, 800, 240, 600)])
    assert 0 < strips - single < 16e6


def test_batches_of_other_parts_in_the_same_buffers():
    rng = np.random.default_rng(32)
    a, b, c = _region(rng, 8, 300, 3000), _region(rng, 40, 520, 600), _region(rng, 8, 300, 700)
    eng, fresh = Engine(), Engine()
    try:
        for regions in ([a, b], [c, b], [b, a], [c, b], [a, c, b]):
            wl = workload.from_pairs(regions)
            for _ in range(2):
                with eng.batch(wl) as kept:
                    kept.forward(native.MODE_FP32_RERUN)
                    got = kept.results()
                with fresh.batch(wl) as new:
                    new.forward(native.MODE_FP32_RERUN)
                    want = new.results()
                fresh.trim()
                assert np.array_equal(got, want)
    finally:
        eng.close()
        fresh.close()
