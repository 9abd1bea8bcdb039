"""Batches of a queue of the default size grow from 1e9 cells, doubling, anew after every flush; a batch size that the
caller names holds from the first batch on.  The results are those of one batch either way."""
import numpy as np
import pytest

from gatk_gb300 import workload as W

pytestmark = pytest.mark.gpu


def _batches(cells, first, most):
    n, open_cells = 0, 0
    for c in cells:
        open_cells += int(c)
        if open_cells >= first:
            n, open_cells, first = n + 1, 0, min(2 * first, most)
    return n + (open_cells > 0)


@pytest.mark.parametrize("which,regions", [(0, 10), (1, 150), (4, 60)])
def test_queue_batches_grow_and_results_match_one_batch(engine, which, regions):
    wl = W.generate(which, regions=regions)
    cells = wl.cells_per_region()
    with engine.batch(wl) as b:
        b.forward()
        want = b.results()
    with engine.queue() as q:
        for k in (1, 2):
            out = q.push(wl)
            q.flush()
            np.testing.assert_array_equal(out, want)
            assert q.info()["n_batches"] == k * _batches(cells, 10**9, 2 * 10**11)
    with engine.queue(batch_cells=4 * 10**9) as q:
        out = q.push(wl)
        q.flush()
        np.testing.assert_array_equal(out, want)
        assert q.info()["n_batches"] == _batches(cells, 4 * 10**9, 4 * 10**9)
