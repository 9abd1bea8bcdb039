"""Contexts opened, used and closed from several threads at once share one pool of host threads and keep one spare batch
each; results stay those of one context used alone."""
import threading

import numpy as np
import pytest

from gatk_gb300 import native, workload
from gatk_gb300.pairhmm import CudaLoglessPairHMM, Engine

pytestmark = pytest.mark.gpu


def test_contexts_in_several_threads():
    wls = [workload.generate(1, regions=12, region_begin=12 * k) for k in range(4)]
    one = Engine()
    want = [one.compute(wl) for wl in wls]
    one.close()
    failed = []

    def work(k):
        try:
            for _ in range(3):
                eng = Engine()
                try:
                    for j in (k, (k + 1) % 4):
                        if not np.array_equal(eng.compute(wls[j]), want[j]):
                            failed.append((k, j))
                finally:
                    eng.close()
        except Exception as e:
            failed.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


@pytest.mark.parametrize("order", [(0, 1, 2, 0), (2, 0, 1, 1)])
def test_batches_one_after_the_other(order):
    """A batch that takes over a destroyed one's buffers, whatever kind that was, starts as a new one."""
    wls = [workload.generate(1, regions=n, region_begin=50) for n in (3, 9, 1)]
    flags = workload.pd_flags(wls[1], 3)
    mapq = [np.full(wl.n_reads, 50) for wl in wls]
    eng = Engine()
    try:
        want = [eng.compute(wl) for wl in wls]
        raw = [eng.compute_raw(wl, mq) for wl, mq in zip(wls, mapq)]
        pd = eng.pd_compute(wls[1], flags)
        for k in order:
            with eng.batch(wls[k]) as b:
                assert b.stats()["ms_total"] == 0 and b.stats()["n_rerun"] == 0
                b.forward()
                assert np.array_equal(b.results(), want[k])
            with eng.raw_batch(wls[k], mapq[k]) as b:
                b.forward()
                assert np.array_equal(b.results(), raw[k])
            with eng.pd_batch(wls[1], flags) as b:
                with pytest.raises(native.GhmmError):
                    b.forward(native.MODE_FP32_RERUN)
                b.forward(native.MODE_PD_FP32)
                assert np.array_equal(b.results(), pd)
    finally:
        eng.close()


def test_plugin_takes_any_byte_sequence():
    haps = [b"ACGTACGTTGCA", b"ACGTACGATGCA"]
    q = [30] * 6
    want = None
    hmm = CudaLoglessPairHMM()
    try:
        hmm.initialize(haps)
        for form in (bytes, bytearray, list, lambda x: np.array(list(x)), lambda x: np.repeat(np.array(list(x), np.uint8), 2)[::2],
                     lambda x: np.array(list(x), np.uint8)[:, None]):
            reads = [tuple(form(x) for x in (b"ACGTAC", q, [45] * 6, [45] * 6, [10] * 6)),
                     tuple(form(x) for x in (b"TTG", q[:3], [45] * 3, [45] * 3, [10] * 3))]
            got = hmm.compute_log10_likelihoods(reads)
            want = got if want is None else want
            assert np.array_equal(got, want) and np.isfinite(got).all()
        with pytest.raises(ValueError):
            hmm.compute_log10_likelihoods([(b"AC", [30], [45], [45], [10])])
        assert hmm.compute_log10_likelihoods([]) is None
    finally:
        hmm.close()
