"""Synchronous calls on either side of the size from which they run as a pipeline of batches (250,000 pairs): a region's
results do not depend on the batch it is in, so both give the bits of one batch, and an argument error stays one."""
import numpy as np
import pytest

from gatk_gb300 import native
from gatk_gb300 import workload as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which,regions", [(3, 31249), (3, 31250), (0, 490), (1, 200)])
def test_calls_around_the_pipelining_size_match_one_batch(engine, which, regions):
    wl = W.generate(which, regions=regions)  # workload 3 has 8 pairs a region: 249,992 and 250,000 pairs
    if which == 3:
        assert wl.n_pairs == 8 * regions
    with engine.batch(wl) as b:
        b.forward()
        want = b.results()
    for via_regions in (True, False):
        np.testing.assert_array_equal(engine.compute(wl, via_regions=via_regions), want)


def test_argument_error_in_the_last_chunk(engine):
    wl = W.generate(3, regions=32000)
    want = engine.compute(wl)
    regs = wl.as_regions()
    last = regs[wl.n_regions - 1].reads[0]
    length, last.length = last.length, 1 << 30
    out = np.zeros(wl.n_pairs)
    rc = engine.L.ghmm_compute_regions(engine._ctx.h, regs, wl.n_regions, out.ctypes.data_as(native._f64p))
    with pytest.raises(native.GhmmError, match="read length out of range"):
        native.check(rc, engine._ctx.h)
    last.length = length
    np.testing.assert_array_equal(engine.compute(wl, via_regions=True), want)
