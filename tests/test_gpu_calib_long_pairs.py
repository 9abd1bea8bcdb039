"""Calibration of pairs whose checkpoints would exceed the scratch limit: fewer of them, with the same results, in place of
fewer warps."""
import ctypes
import time

import numpy as np
import pytest

from gatk_gb300 import native, workload
from gatk_gb300 import calibration as C
from gatk_gb300.pairhmm import Engine

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _set(reads, read_length, hap_length):
    rng = np.random.default_rng(41)
    regions = []
    for _ in range(reads // 16):
        hap = ACGT[rng.integers(0, 4, hap_length)]
        rs = []
        for _ in range(16):
            o = int(rng.integers(0, hap_length - read_length + 1))
            n = read_length
            rs.append((hap[o:o + n], rng.integers(20, 41, n), np.full(n, 45), np.full(n, 45), np.full(n, 10)))
        regions.append(([hap], rs))
    return C.CalibrationSet(workload.from_pairs(regions))


def _backward(e, cs, g, c, precision=0):
    import torch

    ll = torch.empty(cs.n_pairs, dtype=torch.float64, device=cs.device)
    go, gc = torch.zeros_like(g), torch.zeros_like(c)
    b = cs.batch(g, c)
    torch.cuda.synchronize()
    t = time.perf_counter()
    native.check(e.L.ghmm_calib_backward(e.handle, ctypes.byref(b), precision, None, ll.data_ptr(), go.data_ptr(),
                                         gc.data_ptr()), e.handle)
    return time.perf_counter() - t, ll, go, gc


@pytest.mark.parametrize("read_length,hap_length", [(150, 5000), (250, 4500), (600, 4500)])
def test_long_pairs_within_the_limit(monkeypatch, read_length, hap_length):
    """Against 24 GiB, which hold a full grid's checkpoints at every eighth step.  The same values are recomputed from
    either's checkpoints: the repository's bar for FP32 gradients.  The time of the longer segments is about a tenth more
    or less; of a grid cut to fit the shorter ones' checkpoints, 1.75 times for 600 x 4,500."""
    import torch

    cs = _set(1216, read_length, hap_length)
    g, c = (x.detach() for x in cs.position_params(C.default_theta()))
    e = Engine()
    try:
        out = {}
        for limit in (None, 24 << 30):
            if limit:
                monkeypatch.setenv("GHMM_CALIB_SCRATCH_BYTES", str(limit))
            out[limit] = min((_backward(e, cs, g, c) for _ in range(4)), key=lambda r: r[0])
    finally:
        e.close()
    (t4, ll4, go4, gc4), (t24, ll24, go24, gc24) = out[None], out[24 << 30]
    assert torch.allclose(ll4, ll24, rtol=0, atol=1e-3)
    for a, b in ((go4, go24), (gc4, gc24)):
        assert float((a - b).abs().max()) <= 1e-3 * float(b.abs().max())
    assert t4 <= 1.4 * t24, (t4, t24)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("read_length", [100, 256, 300])
def test_both_segment_lengths_at_their_edges(monkeypatch, read_length, precision):
    """Haplotypes of 8 n + 1, of 16 n and of 16 n + 1 steps (31 more than their columns)."""
    import torch

    e = Engine()
    try:
        for hap_length in (801, 802, 809, 810, 817, 818):
            cs = _set(16, read_length, hap_length)
            g, c = (x.detach() for x in cs.position_params(C.default_theta()))
            monkeypatch.delenv("GHMM_CALIB_SCRATCH_BYTES", raising=False)
            _, ll, go, gc = _backward(e, cs, g, c, precision)
            monkeypatch.setenv("GHMM_CALIB_SCRATCH_BYTES", str(8 << 20))
            _, ll2, go2, gc2 = _backward(e, cs, g, c, precision)
            assert torch.allclose(ll, ll2, rtol=0, atol=1e-9 if precision else 1e-3)
            for a, b in ((go, go2), (gc, gc2)):
                assert float((a - b).abs().max()) <= (1e-6 if precision else 1e-3) * float(b.abs().max())
    finally:
        e.close()
