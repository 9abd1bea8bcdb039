"""One-shot PD-HMM calls on either side of the size from which they run in chunks (2e9 cells): a region's results do
not depend on the chunk it is in, so both give the bits of one device-resident batch."""
import numpy as np
import pytest

from gatk_gb300 import native
from gatk_gb300 import workload as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("regions,chunked", [(24, False), (60, True)])
def test_one_shot_pd_calls_match_one_batch(engine, regions, chunked):
    wl = W.generate(1, regions=regions)
    assert (wl.cells() >= 2e9) == chunked
    pd = W.pd_flags(wl, 5)
    with engine.pd_batch(wl, pd) as b:
        b.forward(native.MODE_PD_FP32)
        want = b.results()
    np.testing.assert_array_equal(engine.pd_compute(wl, pd), want)
    mapq = np.full(wl.n_reads, 60)
    with engine.pd_raw_batch(wl, pd, mapq) as b:
        b.forward(native.MODE_PD_FP32)
        want = b.results()
    np.testing.assert_array_equal(engine.pd_compute_raw(wl, pd, mapq), want)
