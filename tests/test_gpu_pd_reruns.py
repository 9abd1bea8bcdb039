"""FP64 reruns of the FP32 PD-HMM pass (a pair per block, strips of 32 rows) against the FP64 oracle, for reads at the
edges of a strip and of a round of four strips and haplotypes around the phases of 16 columns."""
import numpy as np
import pytest

from gatk_gb300 import native
from gatk_gb300 import workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [1, 31, 32, 33, 64, 127, 128, 129, 160, 257, 420]


@pytest.mark.parametrize("hap_len", [1, 15, 16, 17, 31, 33, 48, 113, 240, 611])
def test_pd_reruns_match_the_oracle(engine, hap_len):
    rng = np.random.default_rng(hap_len)
    seq = lambda n: bytes(rng.choice(list(b"ACGT"), size=n).astype(np.uint8))
    reads = []
    for n in LENGTHS:  # unrelated bases at quality 60: about -6.5 a mismatch, so the longer reads underflow 2^120
        reads.append((seq(n), np.full(n, 60), np.full(n, 50), np.full(n, 50), np.full(n, 10)))
    wl = W.from_pairs([([seq(hap_len) for _ in range(3)], reads)])
    pd = W.pd_flags(wl, 7)
    ref = O.pd_compute_workload(wl, pd)
    with engine.pd_batch(wl, pd) as b:
        b.forward(native.MODE_PD_FP32)
        got, n_rerun = b.results(), b.stats()["n_rerun"]
    # a pair below the FP32 pass's threshold, 2^-93 / 2^120 = 10^-64.1, is one the FP64 kernel computed
    deep = ref < -70
    assert n_rerun >= deep.sum()
    assert np.abs(got - ref)[deep].max(initial=0) <= 1e-9
    assert np.abs(got - ref).max() <= 1e-3
