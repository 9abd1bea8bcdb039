"""The chunks of a regular call that runs as a pipeline of batches, against a restatement of the rule."""
import ctypes

import numpy as np

from gatk_gb300 import native


def _library_cuts(cells):
    cells = np.ascontiguousarray(cells, dtype=np.int64)
    out = np.zeros(len(cells) + 2, dtype=np.int64)
    n = ctypes.c_int64(0)
    p = ctypes.POINTER(ctypes.c_int64)
    assert native.lib().ghmm_debug_call_cuts(cells.ctypes.data_as(p), len(cells), out.ctypes.data_as(p), len(out),
                                             ctypes.byref(n)) == 0
    return out[: n.value].tolist()


def _cuts(cells):
    total, ends = int(sum(cells)), np.cumsum(cells)
    cut, target = [0], max(min(total // 8, 8 * 10**9), 1)
    while cut[-1] < len(cells):
        done = int(ends[cut[-1] - 1]) if cut[-1] else 0
        # the first region with which the chunk has its cells
        end = max(int(np.searchsorted(ends, done + target)) + 1, cut[-1] + 1)
        cut.append(end if len(cells) - end >= 8 else len(cells))
        target = min(target * 5 // 2, max(total // 3, 1))
    return cut


def test_chunks():
    assert _library_cuts([10**8] * 100) == [0, 13, 45, 79, 100]  # 1.25e9, 3.125e9, a third
    assert _library_cuts([10**8] * 1000) == [0, 80, 280, 614, 948, 1000]  # 8e9, 2e10, a third
    assert _library_cuts([10**8] * 5) == [0, 5]
    assert _library_cuts([]) == [0]
    rng = np.random.default_rng(6)
    for _ in range(200):
        n = int(rng.integers(1, 3000))
        cells = rng.integers(0, 4, size=n) * rng.integers(1, 1000, size=n) * 10 ** int(rng.integers(3, 9))
        got = _library_cuts(cells)
        assert got == _cuts([int(c) for c in cells])
        assert got[0] == 0 and got[-1] == n and all(a < b for a, b in zip(got, got[1:]))
        assert all(n - c >= 8 for c in got[1:-1])


def test_arguments():
    p = ctypes.POINTER(ctypes.c_int64)
    cells, out, n = np.array([5, -1, 7], dtype=np.int64), np.zeros(8, dtype=np.int64), ctypes.c_int64(0)
    assert native.lib().ghmm_debug_call_cuts(cells.ctypes.data_as(p), 3, out.ctypes.data_as(p), 8, ctypes.byref(n)) != 0
