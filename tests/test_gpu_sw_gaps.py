"""Smith-Waterman tracebacks whose diagonal runs and gaps end around the 32 cells the kernel looks ahead, and end cells
that tie along the last column or the bottom row: cigars and offsets identical to the oracle's."""
import numpy as np
import pytest

from gatk_gb300 import smithwaterman as sw
from oracle import oracle

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 30, 31, 32, 33, 34, 63, 64, 65, 96, 97]


def _check(refs, alts, params, strategy):
    aligner = sw.SmithWatermanCudaAligner()
    try:
        got = aligner.align_many(refs, alts, params, strategy, substring_shortcut=False)
    finally:
        aligner.close()
    off = lambda xs: np.cumsum([0] + [len(x) for x in xs])  # noqa: E731
    ro, ao = off(refs), off(alts)
    ops, start, n_ops, offset = oracle.sw_align_pairs(
        np.concatenate(refs), ro[:-1], np.diff(ro), np.concatenate(alts), ao[:-1], np.diff(ao),
        (params.match_value, params.mismatch_penalty, params.gap_open_penalty, params.gap_extend_penalty), int(strategy),
        False)
    for i in range(len(refs)):
        assert got.offset[i] == offset[i], i
        assert np.array_equal(got.ops(i), ops[start[i]:start[i] + n_ops[i]]), i


@pytest.mark.parametrize("strategy", list(sw.SWOverhangStrategy))
def test_runs_and_gaps_around_the_look_ahead(strategy):
    rng = np.random.default_rng(21)
    base = np.frombuffer(b"ACGT", np.uint8)
    refs, alts = [], []
    for run in LENGTHS:
        for gap in LENGTHS:
            a, b, g = (base[rng.integers(0, 4, n)] for n in (run + 20, run, gap))
            refs += [np.concatenate([a, g, b]), np.concatenate([a, b]), np.concatenate([g, a, g[:gap // 2], b, g])]
            alts += [np.concatenate([a, b]), np.concatenate([a, g, b]), np.concatenate([a, b, g[gap // 2:]])]
    for params in (sw.NEW_SW_PARAMETERS, sw.ALIGNMENT_TO_BEST_HAPLOTYPE_SW_PARAMETERS, sw.SWParameters(3, -1, -4, 0)):
        _check(refs, alts, params, strategy)


@pytest.mark.parametrize("strategy", list(sw.SWOverhangStrategy))
def test_tied_end_cells(strategy):
    """One-letter sequences: every cell of a diagonal ties with the next one's."""
    refs, alts = [], []
    for n in (1, 31, 32, 33, 70, 300):
        for m in (1, 31, 32, 33, 64, 65, 130, 260):
            refs.append(np.full(n, 65, np.uint8))
            alts.append(np.full(m, 65, np.uint8))
            alt = np.full(m, 65, np.uint8)
            alt[m // 2:] = 67
            refs.append(np.full(n, 65, np.uint8))
            alts.append(alt)
    for params in (sw.ORIGINAL_DEFAULT, sw.SWParameters(0, 0, 0, 0), sw.SWParameters(1, -1, 0, 0)):
        _check(refs, alts, params, strategy)
