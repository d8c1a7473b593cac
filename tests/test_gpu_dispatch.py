"""The full-DP launch rules on either side of their edges, against the FP64
oracle and against forced unit sizes (bit for bit)."""
import numpy as np
import pytest

from biovoltron_b200 import workloads as W
from oracle.oracle import TestcaseArray

pytestmark = pytest.mark.gpu

TOL_FP32 = 1e-4  # FP32 rounding against 64 bits, as the parity tests allow


def _region(rng, n_reads, n_haps, read_lens, hap_len):
    base = W._random_seq(rng, hap_len)
    haps = [W._apply_indels(rng, W._substitute(rng, base, 0.01), k % 3, 1, 8) for k in range(n_haps)]
    reads = []
    for k in range(n_reads):
        src = haps[k % n_haps]
        n = min(int(read_lens[k % len(read_lens)]), len(src))
        at = int(rng.integers(0, len(src) - n + 1))
        r = W._substitute(rng, src[at:at + n], 0.01)
        reads.append((r, *W._quals(rng, n, 10, 40)))
    return reads, haps


# pairs on either side of half the resident warps (148 SMs x 16 / 2 = 1184: one haplotype a unit or two),
# a single pair, an odd haplotype count, and reads of every bin and of two strips in one batch
@pytest.mark.parametrize("n_reads,n_haps,lens", [(1, 1, [1]), (37, 32, [90, 150]), (79, 15, [29, 30, 61, 62, 150]),
                                                 (60, 33, [29, 30, 61, 93, 125, 157, 189, 221, 253, 254, 300])])
def test_unit_sizes_and_lanes(engine, oracle, n_reads, n_haps, lens):
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(n_reads * 100 + n_haps)
    b = W._build([_region(rng, n_reads, n_haps, lens, 380)], "dispatch")
    got = engine.compute_regions(b)
    truth = oracle.log10_rescaled(TestcaseArray.for_batch(b))
    assert np.max(np.abs(got - truth)) <= TOL_FP32
    for unit, warp in ((32, 2), (1, 1)):
        with PairHMMEngine(haps_per_unit=unit, haps_per_warp=warp) as e:
            assert np.array_equal(e.compute_regions(b), got)
            n = e.stage(b)
            for _ in range(3):  # direct launches, then the captured graph with its parallel branches
                e.run()
                assert np.array_equal(e.fetch(n), got)


# units made on the device (batches over 512 KB of inputs) against those the host fills (small ones): regions
# without reads or haplotypes, read counts around a warp, haplotype counts around a unit, every bin
@pytest.mark.parametrize("precision,band", [("auto", False), ("f64", False), ("auto", True)])
def test_units_made_on_the_device(precision, band):
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(12)
    lens = [1, 29, 30, 61, 62, 94, 125, 126, 157, 158, 190, 222, 252, 253, 254, 300]
    regions = []
    for k in range(160):
        nr, nh = (0, 1, 31, 32, 33, 70)[k % 6], (0, 1, 2, 7, 8, 9, 17)[k % 7]
        reads, haps = _region(rng, nr, max(nh, 1), np.roll(lens, k), 330)
        regions.append((reads, haps[:nh]))
    b = W._build(regions, "units")
    assert b.nbytes() > 1 << 20
    with PairHMMEngine(precision=precision) as e:
        if band:
            e.set_band_options(enabled=True, cap_margin=0)
        got = e.compute_regions(b)
        parts = [W.subsample_regions(b, range(g, g + 8)) for g in range(0, 160, 8)]
        assert all(5 * p.read_bases.size + p.hap_bases.size < 400_000 for p in parts)
        assert np.array_equal(got, np.concatenate([e.compute_regions(p) for p in parts]))
        n = e.stage(b)
        for _ in range(2):
            e.run()
            assert np.array_equal(e.fetch(n), got)


# one haplotype a warp (few pairs) against two, bit for bit: rows that cannot be folded (indel qualities of 0-3),
# N in reads and haplotypes, haplotypes of one base and shorter than the read, every bin's longest read
@pytest.mark.parametrize("gap", [45, 2, 0])
def test_one_haplotype_a_warp(oracle, gap):
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(40 + gap)
    regions = []
    for n in (1, 29, 61, 93, 125, 157, 189, 221, 253):
        reads, haps = _region(rng, 2, 3, [n], n + 40)
        reads = [(r, q, np.full(len(r), gap, np.uint8), np.full(len(r), gap, np.uint8), c) for r, q, _, _, c in reads]
        reads[0][0][len(reads[0][0]) // 2] = ord("N")
        haps[1][5:7] = ord("N")
        regions.append((reads, haps + [haps[0][:1].copy(), haps[0][:n // 2 + 1].copy()]))
    b = W._build(regions, "one haplotype a warp")
    out = []
    for warp in (1, 2):
        with PairHMMEngine(haps_per_unit=4, haps_per_warp=warp) as e:
            out.append(e.compute_regions(b))
    assert np.array_equal(out[0], out[1])
    truth = oracle.log10_rescaled(TestcaseArray.for_batch(b))
    fin = np.isfinite(truth)
    assert np.array_equal(np.isfinite(out[0]), fin)
    assert np.max(np.abs(out[0][fin] - truth[fin])) <= TOL_FP32


# reads of several strips that stay in FP32, at the strips' edges (256 rows, the initial and the summing row among
# them), haplotypes shorter than a 32-column chunk and around its multiples, rows that cannot be folded
@pytest.mark.parametrize("gap", [45, 2])
@pytest.mark.parametrize("read_len", [254, 255, 256, 510, 511, 512, 766, 767])
def test_strips(oracle, read_len, gap):
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(read_len + gap)
    regions = []
    for hap_len in (read_len, read_len + 1, read_len + 31, read_len + 32, read_len + 33, read_len + 200):
        hap = W._random_seq(rng, hap_len)
        q, i, d, c = W._quals(rng, read_len, 40, 45)
        i, d = np.full(read_len, gap, np.uint8), np.full(read_len, gap, np.uint8)
        regions.append(([(hap[:read_len].copy(), q, i, d, c)], [hap, hap[:read_len].copy(), hap[:20].copy()]))
    b = W._build(regions, "strips")
    truth = oracle.log10_rescaled(TestcaseArray.for_batch(b))
    with PairHMMEngine() as e:
        got, st = e.compute_regions(b, with_stats=True)
        assert np.max(np.abs(got - truth)) <= TOL_FP32
        if gap == 45:  # the reads match: only the haplotypes of 20 bases need FP64
            assert st["rescued"] <= len(regions)


def test_set_shapes_in_a_small_batch():
    """A small batch with shapes set for its bin, for another bin, for all of them, one or two haplotypes a warp: the
    same values; haplotypes too long for two a warp are accepted either way."""
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(50)
    batches = [W._build([_region(rng, 64, 8, [150], 300)], "window"), W._build([_region(rng, 2, 3, [150], 20000)], "long")]
    out = []
    for bins, haps in (((), 2), ((3,), 2), ((5,), 2), (range(1, 9), 2), (range(1, 9), 1)):
        with PairHMMEngine() as e:
            e.set_tuning([{"rows_per_lane": rt, "haps_per_warp": haps, "warps_per_block": 2} for rt in bins])
            out.append([e.compute_regions(b) for b in batches])
    for o in out[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(o, out[0]))
