"""FP64 lists of short and long reads: the long reads' pairs a block each, the others' a warp each, both tiers, any
order in the list; and the short ones at their own speed."""
import numpy as np
import pytest

from gatk_gb300 import native, workload
from gatk_gb300.pairhmm import Engine
from oracle import oracle

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _region(rng, read_lengths, hap_lengths, ins=(30, 46)):
    reads = [(ACGT[rng.integers(0, 4, n)], rng.integers(6, 41, n), rng.integers(*ins, n), rng.integers(*ins, n),
              np.full(n, 10)) for n in read_lengths]
    return [ACGT[rng.integers(0, 4, n)] for n in hap_lengths], reads


def _agrees(got, want, bar=1e-9):  # the repository's bar for FP64 results
    differ = got != want  # (infinities are equal)
    return np.max(np.abs(got[differ] - want[differ]), initial=0.0) <= bar


@pytest.mark.parametrize("ins", [(30, 46), (3, 4)], ids=["rescaled_tier", "exact_tier"])
@pytest.mark.parametrize("long_reads", [[481], [480, 481, 482, 513], [600] * 12], ids=str)
def test_double_precision(long_reads, ins):
    """More pairs than any grid has warps, the long reads in some of the regions, haplotypes empty and of a phase's edges."""
    rng = np.random.default_rng(51)
    short = [1, 31, 32, 33, 64, 100, 128, 129, 161, 256, 257, 385]
    haps = [1, 16, 17, 0, 48, 97, 130, 3, 3, 210]
    regions = [_region(rng, short, haps, ins) for _ in range(30)]
    regions[3:3] = [_region(rng, short[:4] + long_reads + short[4:], haps + [640], ins)]
    regions.append(_region(rng, long_reads, [700, 5], ins))
    wl = workload.from_pairs(regions)
    assert wl.n_pairs > 3000
    eng = Engine(use_double_precision=True)
    try:
        with eng.batch(wl) as b:
            for _ in range(2):  # launched, then captured
                b.forward(native.MODE_FP64)
                assert _agrees(b.results(), oracle.compute_workload(wl))
    finally:
        eng.close()


def test_reruns_of_an_fp32_pass():
    """Every second pair forced into FP64, in the order the FP32 pass queues them, beside pairs that are routed there."""
    wl = workload.generate(1, regions=16)
    rng = np.random.default_rng(52)
    regions = [([wl.hap(h) for h in range(int(wl.region_hap_off[g]), int(wl.region_hap_off[g + 1]))],
                [wl.read(r) for r in range(int(wl.region_read_off[g]), int(wl.region_read_off[g + 1]))])
               for g in range(16)]
    regions.append(_region(rng, [481, 100, 700], [500, 900]))
    wl = workload.from_pairs(regions)
    eng = Engine()
    try:
        native.check(eng.L.ghmm_debug_inject(eng.handle, native.INJECT_FP64_RERUN_EVERY, 2), eng.handle)
        with eng.batch(wl) as b:
            b.forward(native.MODE_FP32_RERUN)
            got, n = b.results(), b.stats()["n_rerun"] + b.stats()["n_fp64_direct"]
    finally:
        eng.L.ghmm_debug_inject(eng.handle, native.INJECT_FP64_RERUN_EVERY, 0)
        eng.close()
    want = oracle.compute_workload(wl)
    assert n > 3000 and _agrees(got[::2], want[::2])
    assert _agrees(got, want, 1e-3)


def test_one_long_read_among_short_ones_costs_its_own_time():
    """40,960 pairs of 30 x 300 bases, and one of 481 x 600: with every pair a block each they take three times as long.
    The sum of the two apart, and a quarter."""
    rng = np.random.default_rng(53)
    short = [_region(rng, [30] * 40, [300] * 16) for _ in range(64)]
    one = [_region(rng, [481], [600])]
    ms = {}
    eng = Engine(use_double_precision=True)
    try:
        for name, regions in (("short", short), ("one", one), ("both", short + one)):
            with eng.batch(workload.from_pairs(regions)) as b:
                times = []
                for _ in range(6):
                    b.forward(native.MODE_FP64)
                    times.append(b.stats()["ms_fp64"])
                ms[name] = min(times)
    finally:
        eng.close()
    assert ms["both"] <= 1.25 * (ms["short"] + ms["one"]), ms
