"""Errors of synchronous calls that run as several batches are those of one batch: an input error leaves the caller's
array as it was, wherever the bad read is, and an invalid result is named by its place in that array, the others being
there."""
import ctypes
import re

import numpy as np
import pytest

from gatk_gb300 import native
from gatk_gb300 import workload as W
from gatk_gb300.pairhmm import _read_prep

pytestmark = pytest.mark.gpu

REGIONS = 32000  # of workload 3: 8 pairs each, 256,000 in all


def _workload():
    return W.generate(3, regions=REGIONS).subset(0, REGIONS)  # (a copy)


def _call(engine, wl, form, out):
    p = out.ctypes.data_as(native._f64p)
    if form == "regions":
        return engine.L.ghmm_compute_regions(engine.handle, wl.as_regions(), wl.n_regions, p)
    if form == "flat":
        f = wl.as_flat()
        return engine.L.ghmm_compute_flat(engine.handle, ctypes.byref(f), p)
    prep = _read_prep(18, True, 3.0, 10, None, wl)
    regs = W.as_raw_regions(wl, np.full(wl.n_reads, 50), True)
    return engine.L.ghmm_compute_regions_raw(engine.handle, regs, wl.n_regions, ctypes.byref(prep), p)


@pytest.mark.parametrize("form", ["regions", "flat", "raw"])
@pytest.mark.parametrize("where", [0.0, 0.3, 0.6, 1.0])
def test_input_error_leaves_the_array(engine, form, where):
    wl = _workload()
    wl.quals[int(where * (len(wl.quals) - 1))] = 255
    out = np.full(wl.n_pairs, 7.0)
    with pytest.raises(native.GhmmError, match="quality out of range"):
        native.check(_call(engine, wl, form, out), engine.handle)
    assert (out == 7.0).all()


def test_invalid_results(engine):
    """Insertion and deletion penalties of 0 make the transitions' probabilities sum to more than 1; a read and a
    haplotype of one repeated base then grow without bound."""
    good = _workload()
    want = engine.compute(good)
    for regions in ([0], [REGIONS // 2], [REGIONS - 1], [5, REGIONS // 3, REGIONS - 3]):
        wl = _workload()
        bad = np.zeros(wl.n_pairs, bool)
        for g in regions:
            r = int(wl.region_read_off[g])
            a, b = int(wl.read_off[r]), int(wl.read_off[r + 1])
            wl.ins[a:b] = wl.dels[a:b] = 0
            h = int(wl.region_hap_off[g])
            wl.bases[a:b] = wl.hap_bases[int(wl.hap_off[h]):int(wl.hap_off[h + 1])] = ord("A")
            bad[int(wl.out_off[g]):int(wl.out_off[g + 1])] = True  # (the region's other reads are valid, but others)
        for form in ("regions", "flat"):
            out = np.full(wl.n_pairs, 7.0)
            with pytest.raises(native.GhmmError, match="not a valid log10 probability") as err:
                native.check(_call(engine, wl, form, out), engine.handle)
            assert err.value.code == native.GHMM_ERR_RESULT
            place = int(re.search(r"at output (\d+) is", str(err.value)).group(1))
            assert place in wl.out_off[regions] and not out[place] <= 0
            assert np.array_equal(out[~bad], want[~bad])
