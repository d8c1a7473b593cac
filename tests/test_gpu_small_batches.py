"""Batches on either side of the size that is staged as one page-locked image
(512 KB of inputs) and of the results that come back with the counters (32,768):
the same values, whatever the gap penalties' form, alone and after one another."""
import numpy as np
import pytest

from biovoltron_b200 import workloads as W
from oracle.oracle import TestcaseArray

pytestmark = pytest.mark.gpu


def _batch(n_reads, n_haps, read_len, hap_len, seed, varied):
    rng = np.random.default_rng(seed)
    base = W._random_seq(rng, hap_len)
    haps = [W._substitute(rng, base, 0.01) for _ in range(n_haps)]
    reads = []
    for k in range(n_reads):
        n = max(1, read_len - k % 17)
        at = int(rng.integers(0, hap_len - n + 1))
        r = W._substitute(rng, haps[k % n_haps][at:at + n], 0.01)
        q, i, d, c = W._quals(rng, n, 10, 40)
        if varied:
            i, d, c = (rng.integers(20, 50, n).astype(np.uint8) for _ in range(3))
        reads.append((r, q, i, d, c))
    return W._build([(reads, haps)], "small")


# reads x haplotypes: tiny; image just under and over 512 KB; results just under, at and over 32,768
@pytest.mark.parametrize("shape", [(1, 1, 17, 40), (5, 3, 33, 60), (640, 2, 150, 200), (800, 2, 150, 200),
                                   (1024, 31, 60, 90), (1024, 32, 60, 90), (1025, 32, 60, 90)])
@pytest.mark.parametrize("varied", [False, True])
def test_sizes_around_the_image(engine, oracle, shape, varied):
    b = _batch(*shape, seed=shape[0], varied=varied)
    got = engine.compute_regions(b)
    n = engine.stage(b)
    for _ in range(2):
        engine.run()
        assert np.array_equal(engine.fetch(n), got)
    if not varied:
        assert np.array_equal(engine.compute_regions(b, uniform_gaps=(45, 45, 10)), got)
    r, h = b.pair_index()
    pick = np.random.default_rng(1).choice(b.n_pairs, min(b.n_pairs, 300), replace=False)
    truth = oracle.log10_rescaled(TestcaseArray(b, r[pick], h[pick]))
    assert np.max(np.abs(got[pick] - truth)) <= 1e-4  # FP32 rounding, as the parity tests allow


def test_small_and_large_in_turn(engine):
    """One context, a small batch after a large one and back: buffers that were views are allocations again."""
    small, large = _batch(20, 3, 100, 200, 3, True), _batch(1200, 32, 100, 200, 4, True)
    a, b = engine.compute_regions(small), engine.compute_regions(large)
    for _ in range(2):
        assert np.array_equal(engine.compute_regions(small), a)
        assert np.array_equal(engine.compute_regions(large), b)
    engine.set_band_options(enabled=True)
    try:
        c = engine.compute_regions(small)
        assert np.max(np.abs(c - a)) <= 1e-3
        engine.compute_regions(large)
        assert np.array_equal(engine.compute_regions(small), c)
    finally:
        engine.set_band_options(enabled=False)
    assert np.array_equal(engine.compute_regions(small), a)


def test_launches_are_counted(engine):
    """One bin: its kernel, the FP64 list's, and a small batch's copy back; a larger batch's staging makes the units and
    packs the qualities."""
    for n_reads, staging in ((20, 0), (1200, 2)):
        b = _batch(n_reads, 8, 150, 300, 5, False)
        _, st = engine.compute_regions(b, with_stats=True)
        run = 2 + (staging == 0)
        assert st["kernel_launches"] == run + staging
        engine.stage(b)
        assert engine.run()["kernel_launches"] == run
