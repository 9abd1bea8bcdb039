"""The buffers a context keeps of its last destroyed batch: given back on request, and to an allocation that finds no
memory."""
import numpy as np
import pytest

from gatk_gb300 import native, workload
from gatk_gb300.pairhmm import Engine

pytestmark = pytest.mark.gpu


def _keep_one(eng, wl):
    with eng.batch(wl) as b:
        b.forward()
        return b.results()


def test_trim_gives_the_kept_buffers_back():
    wl = workload.generate(1, regions=3)
    eng = Engine()
    try:
        assert eng.trim() == 0
        want = _keep_one(eng, wl)
        assert eng.trim() > wl.n_pairs * 8
        assert eng.trim() == 0
        assert np.array_equal(_keep_one(eng, wl), want)
    finally:
        eng.close()


def test_an_allocation_without_memory_takes_the_kept_buffers():
    small, large = workload.generate(1, regions=2), workload.generate(1, regions=9)
    a, b = Engine(), Engine()
    try:
        want = b.compute(large)
        _keep_one(a, small)
        native.check(b.L.ghmm_debug_inject(b.handle, native.INJECT_FULL_MEMORY, 1), b.handle)
        assert np.array_equal(_keep_one(b, large), want)
        assert a.trim() == 0  # (b's batch had it)
        # nothing kept any more: the call fails, and the context stays usable
        b.trim()
        native.check(b.L.ghmm_debug_inject(b.handle, native.INJECT_FULL_MEMORY, 2), b.handle)
        with pytest.raises(native.GhmmError) as err:
            b.batch(large)
        assert err.value.code == native.GHMM_ERR_NOMEM
        native.check(b.L.ghmm_debug_inject(b.handle, native.INJECT_FULL_MEMORY, 0), b.handle)
        assert np.array_equal(_keep_one(b, large), want)
    finally:
        b.L.ghmm_debug_inject(b.handle, native.INJECT_FULL_MEMORY, 0)
        a.close()
        b.close()


def test_constant_matches_the_header():
    import os
    import re

    hdr = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "include", "ghmm.h")).read()
    assert int(re.search(r"#define GHMM_INJECT_FULL_MEMORY (\d+)", hdr).group(1)) == native.INJECT_FULL_MEMORY
