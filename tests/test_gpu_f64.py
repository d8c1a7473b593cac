"""FP64 kernels in the scaled, folded form (single strips, long reads) at the
edges of their range, against the rescaled FP64 oracle: |d log10| <= 1e-9, the
bound the unscaled FP64 kernels are held to."""
import numpy as np
import pytest

from biovoltron_b200 import workloads as W
from oracle.oracle import TestcaseArray

pytestmark = pytest.mark.gpu

TOL = 1e-9


def _check(b, got, oracle):
    truth = oracle.log10_rescaled(TestcaseArray.for_batch(b))
    fin = np.isfinite(truth)
    assert np.array_equal(np.isfinite(got), fin)
    assert np.max(np.abs(got[fin] - truth[fin]), initial=0) <= TOL


def _pair(rng, n, hap_len, related=True, gaps=(45, 45, 10), qlo=10, qhi=40):
    hap = W._random_seq(rng, hap_len)
    at = int(rng.integers(0, max(1, hap_len - n + 1)))
    read = W._mutate_read(rng, hap, at, n, 0.02, 0.01, 1, 3) if related and hap_len >= n else W._random_seq(rng, n)
    q, i, d, c = W._quals(rng, len(read), qlo, qhi, *gaps)
    return [(read, q, i, d, c)], [hap]


# every rows-per-lane bin's edges, the longest single strip (253) and the first two-strip reads, haplotypes
# shorter and longer than the read, unrelated pairs (results far below the kept range: handed to the
# unscaled kernel), rows that cannot fold (indel qualities of 0-3), varying gap qualities
def _short_cases(rng):
    regions = []
    for n in (1, 2, 28, 29, 30, 61, 62, 93, 94, 125, 126, 157, 158, 189, 190, 221, 222, 252, 253, 254, 255, 300):
        regions.append(_pair(rng, n, n + int(rng.integers(0, 200))))
        regions.append(_pair(rng, n, 3 + n // 2, related=False))
    for n in (150, 253):
        regions.append(_pair(rng, n, 400, related=False, qlo=39, qhi=40))
        regions.append(_pair(rng, n, 400, gaps=(2, 2, 10)))
        regions.append(_pair(rng, n, 400, gaps=(0, 3, 0)))
    reads, haps = _pair(rng, 200, 500)
    r, q, i, d, c = reads[0]
    i, d, c = (rng.integers(0, 128, len(r)).astype(np.uint8) for _ in range(3))
    regions.append(([(r, q, i, d, c), (r, q, i | 16, d | 16, c)], haps * 3))
    return W._build(regions, "short reads in FP64")


def test_single_strip_edges(oracle):
    from biovoltron_b200.pairhmm import PairHMMEngine
    b = _short_cases(np.random.default_rng(3))
    with PairHMMEngine(precision="f64") as e:
        got, st = e.compute_regions(b, with_stats=True)
        _check(b, got, oracle)
        assert st["rescued"] == b.n_pairs and st["rescued_cells"] == b.n_cells()
        n = e.stage(b)
        for _ in range(3):  # the handed-back pairs are scored again by every replay
            e.run()
            assert np.array_equal(e.fetch(n), got)
    with PairHMMEngine() as e:  # the rescue of the pairs FP32 cannot hold takes the same kernels
        auto, st = e.compute_regions(b, with_stats=True)
        assert 0 < st["rescued"] < b.n_pairs
        fin = np.isfinite(got)
        assert np.all(np.abs(auto[fin] - got[fin]) <= 1e-4)


def test_units_of_several_haplotypes(oracle):
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(5)
    b = W.config1(seed=11, n_regions=3)
    out = []
    for unit in (1, 3, 8):
        with PairHMMEngine(precision="f64", haps_per_unit=unit) as e:
            out.append(e.compute_regions(b))
    _check(b, out[0], oracle)
    assert all(np.array_equal(o, out[0]) for o in out)


def test_scalar_transitions_with_a_zero(engine, oracle):
    """A zero insertion probability has no scaled form: the unscaled kernel takes the pair."""
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(7)
    b = W._build([_pair(rng, 120, 260), _pair(rng, 700, 900)], "scalar")
    for trans in ((0.9998, 0.0001, 0.0001, 0.9, 0.1, 0.9, 0.1), (0.9999, 0.0, 0.0001, 0.9, 0.1, 0.9, 0.1)):
        with PairHMMEngine(precision="f64") as e:
            e.set_transitions(trans)
            got = e.compute_regions(b)
        for k in range(b.n_reads):
            rd = b.read(k)
            want = oracle.scalar_log10(bytes(rd[0]), bytes(rd[1]), b.hap(k), trans)
            if np.isfinite(want):
                assert abs(got[k] - want) <= TOL


# strip and group edges of the long-read kernel; few pairs (clusters of four and two blocks of 16 warps, one
# round of them and two), more pairs (one block a pair), unrelated pairs whose mass falls by thousands of binary orders, a read longer
# than its haplotype, rows that cannot fold
@pytest.mark.parametrize("copies", [1, 3, 5, 9, 18])
def test_long_reads(oracle, copies):
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(9)
    regions = [_pair(rng, n, h) for n, h in ((254, 300), (255, 700), (256, 256), (383, 500), (511, 640), (512, 900),
                                             (1023, 1100), (1024, 1300), (2047, 2100), (2048, 2300), (2049, 2200),
                                             (4095, 4200), (4500, 5000))]
    regions += [_pair(rng, 900, 600, related=False), _pair(rng, 1500, 1500, related=False, qlo=38, qhi=40),
                _pair(rng, 2500, 3000, gaps=(20, 60, 10)), _pair(rng, 300, 33, related=False), _pair(rng, 400, 1),
                _pair(rng, 600, 900, gaps=(1, 2, 10))]
    b = W._build(regions, "long reads")
    big = W._build(regions * copies, "long reads, several times")
    with PairHMMEngine(precision="f64") as e:
        got = e.compute_regions(big)
        assert np.array_equal(got.reshape(copies, -1), np.tile(got[:b.n_pairs], (copies, 1)))
        _check(b, got[:b.n_pairs], oracle)
        n = e.stage(big)
        for _ in range(2):
            e.run()
            assert np.array_equal(e.fetch(n), got)
        for k in (2, 4, 8):
            e.set_long_warps(k)
            _check(b, e.compute_regions(b), oracle)
    with PairHMMEngine() as e:
        _, st = e.compute_regions(b, with_stats=True)
        assert st["rescued"] > 0


def test_long_read_on_eight_blocks(oracle):
    """Reads of more strips than four blocks have warps, and the strip counts around eight blocks' 128."""
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(10)
    b = W._build([_pair(rng, n, h) for n, h in ((16383, 1200), (16384, 900), (16500, 700), (8300, 8400), (254, 300))],
                 "very long reads")
    with PairHMMEngine(precision="f64") as e:
        got = e.compute_regions(b)
        _check(b, got, oracle)
        assert np.array_equal(e.compute_regions(b), got)


def test_longest_haplotypes(oracle):
    """The longest haplotypes that are accepted: a block's four of them and the emission tables of seven and eight rows a lane."""
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(12)
    b = W._build([_pair(rng, n, 32768) for n in (100, 157, 190, 253)], "long haplotypes")
    with PairHMMEngine(precision="f64") as e:
        _check(b, e.compute_regions(b), oracle)


@pytest.mark.parametrize("pairs", [100, 512, 513])
def test_long_reads_of_very_different_lengths(oracle, pairs):
    """Cluster launches of every size side by side (a few long reads among many short ones), up to the most pairs
    they take and one more."""
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(13)
    some = [_pair(rng, n, n + 100) for n in (6000, 4100, 2300, 1000, 520, 254, 300)]
    some.append(_pair(rng, 3000, 900, related=False))
    regions = some + [some[4 + k % 3] for k in range(pairs - len(some))]
    b = W._build(regions, "very different lengths")
    with PairHMMEngine(precision="f64") as e:
        got = e.compute_regions(b)
        first = W._build(some, "one of each")
        _check(first, got[:len(some)], oracle)
        assert np.array_equal(got[len(some):], np.array([got[4 + k % 3] for k in range(pairs - len(some))]))
        n = e.stage(b)
        for _ in range(3):
            e.run()
            assert np.array_equal(e.fetch(n), got)


def _strip_bases(n, strip):
    """The read bases [a, b) whose rows the long-read kernel's strip holds (128 rows, row 0 and the padding on top)."""
    pad = -(n + 1) % 128
    return max(0, 128 * strip - pad - 1), 128 * (strip + 1) - pad - 1


def _blocked(rng, n, q, gcp, strips, rival):
    """A read of A and C; a haplotype that is the read but for whole strips of other bases, so that a path along it
    loses 1,000 to 1,600 binary orders within a strip; with `rival` a second copy behind it that loses 600 to 800 in
    each of two strips, so that the lower of two paths after one strip is the better one after both."""
    read = rng.choice(np.frombuffer(b"AC", np.uint8), n)
    first = read.copy()
    for s in strips:
        a, b = _strip_bases(n, s)
        first[a:b] = rng.choice(np.frombuffer(b"GT", np.uint8), b - a)
    hap = [W._random_seq(rng, 40), first, W._random_seq(rng, 40)]
    if rival:
        second = read.copy()
        for s in (strips[0], strips[0] + 1):
            a, b = _strip_bases(n, s)
            at = a + rng.choice(b - a, 70, replace=False)
            second[at] = rng.choice(np.frombuffer(b"GT", np.uint8), 70)
        hap.append(second)
    q, i, d, c = W._quals(rng, n, q, q, gcp=gcp)
    return [(read, q, i, d, c)], [np.concatenate(hap)]


# strips whose rows cost more than half of FP64's exponent range (a stretch of the read that does not align and
# insertion runs too dear to bridge it), read lengths of three, five and twenty strips, the second and the last but one
# of them, or two at once; one path, or two of which the one that is lower after the strip wins in the end
@pytest.mark.parametrize("rival", [False, True])
@pytest.mark.parametrize("n", [300, 600, 2500])
def test_long_reads_that_lose_most_of_the_range_in_a_strip(oracle, n, rival):
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(n)
    last = (n + 1 + 127) // 128 - 1
    regions = [_blocked(rng, n, q, gcp, strips, rival)
               for q, gcp in ((25, 40), (26, 30), (28, 45), (30, 40), (30, 60))
               for strips in ([1], [last - 1], [last - 1] if rival else [1, last])]
    if n <= 600:  # a read that belongs to nothing in a short haplotype
        regions.append(_pair(rng, n, 180, related=False, gaps=(45, 45, 30), qlo=30, qhi=34))
    b = W._build(regions, "range within a strip")
    for precision in ("f64", "auto"):  # every pair in FP64, and the rescue
        with PairHMMEngine(precision=precision) as e:
            got, st = e.compute_regions(b, with_stats=True)
            assert st["rescued"] == b.n_pairs
            _check(b, got, oracle)
            for k in (2, 4, 8):
                if n >= 128 * k:  # the long-read kernel's edge
                    e.set_long_warps(k)
                    _check(b, e.compute_regions(b), oracle)


@pytest.mark.parametrize("gcp", [30, 40, 60])
def test_long_reads_with_dear_gaps(oracle, gcp):
    """Reads of up to 10 kb whose insertion runs cost 10 to 20 binary orders a base: far from the alignment nothing stays
    in range, and a strip's scale has to follow the row above when the alignment comes back, thousands of binary orders
    away.  Insertion qualities of one value, and jumping between rows."""
    from dataclasses import replace
    from biovoltron_b200.pairhmm import PairHMMEngine
    b = W.config2(seed=40, n_pairs=12)
    rng = np.random.default_rng(gcp)
    b = replace(b, read_c=np.full_like(b.read_c, gcp))
    for b in (b, replace(b, read_i=rng.integers(8, 46, b.read_i.size).astype(np.uint8))):
        with PairHMMEngine(precision="f64") as e:
            _check(b, e.compute_regions(b), oracle)
            for k in (2, 8):
                e.set_long_warps(k)
                _check(b, e.compute_regions(b), oracle)


# indel qualities whose pMM is small: the smallest that is positive (1 and 7: 0.006), zero (not folded), and both among
# others; single strips, the list, long reads
@pytest.mark.parametrize("gaps", [(1, 7, 10), (5, 2, 20), (4, 4, 10), (1, 6, 10), (0, 127, 30)])
def test_rows_with_a_small_match_probability(oracle, gaps):
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(sum(gaps))
    regions = []
    for n in (60, 150, 253, 254, 700, 1500):
        for related in (True, False):
            reads, haps = _pair(rng, n, n + 150, related=related, gaps=gaps)
            r, q, i, d, c = reads[0]
            some = rng.random(len(r)) < 0.3
            regions.append((reads + [(r, q, np.where(some, i, 40).astype(np.uint8), np.where(some, d, 45).astype(np.uint8), c)],
                            haps))
    b = W._build(regions, "small pMM")
    with PairHMMEngine(precision="f64") as e:
        _check(b, e.compute_regions(b), oracle)


def test_constant_transitions_that_lose_most_of_the_range_in_a_strip(oracle):
    """Insertion runs that are dear by a small insertion-to-insertion probability."""
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(17)
    b = W._build([_blocked(rng, 300, q, 10, [1], False) for q in (25, 28, 30)], "scalar, range within a strip")
    trans = (0.9998, 0.0001, 0.0001, 0.999999, 0.000001, 0.9, 0.1)
    with PairHMMEngine(precision="f64") as e:
        e.set_transitions(trans)
        got = e.compute_regions(b)
    want = [oracle.scalar_log10(bytes(b.read(k)[0]), bytes(b.read(k)[1]), b.hap(k), trans) for k in range(b.n_reads)]
    assert np.max(np.abs(got - want)) <= TOL


# the unscaled strips, which reads below the long-read kernel's edge take (512 bases with 4 warps, 1,024 with 8) and
# pairs that other kernels hand back: a row between two strips below 2^-24 needs a factor of more than 2^1023
@pytest.mark.parametrize("n", [300, 600])
def test_unscaled_strips_that_lose_most_of_the_range(oracle, n):
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(n)
    regions = [_blocked(rng, n, q, gcp, strips, False) for q, gcp in ((15, 30), (20, 30), (25, 40), (28, 45), (30, 60))
               for strips in ([1], [1, (n + 128) // 128 - 1])]
    regions += [_pair(rng, n, 180, related=False, gaps=(45, 45, gcp), qlo=30, qhi=34) for gcp in (20, 25, 30)]
    b = W._build(regions, "unscaled strips")
    with PairHMMEngine(precision="f64") as e:
        e.set_long_warps(8)
        _check(b, e.compute_regions(b), oracle)


def _hopeless(rng):
    """Reads that lose more than 2,000 binary orders in 128 rows: bases of one kind against haplotypes of another, with
    insertion runs as dear as mismatches."""
    regions = []
    for n, q, gcp in ((200, 55, 70), (254, 50, 60), (300, 48, 60), (600, 50, 50), (900, 60, 70)):
        read = rng.choice(np.frombuffer(b"AC", np.uint8), n)
        qs, i, d, c = W._quals(rng, n, q, q, gcp=gcp)
        regions.append(([(read, qs, i, d, c)], [rng.choice(np.frombuffer(b"GT", np.uint8), h) for h in (n // 3, n + 70)]))
    return W._build(regions, "hopeless reads")


def test_strips_that_lose_more_than_the_range(oracle):
    """What no strip of 128 rows holds is scored in strips of 32."""
    from biovoltron_b200.pairhmm import PairHMMEngine
    b = _hopeless(np.random.default_rng(19))
    for precision in ("f64", "auto"):
        with PairHMMEngine(precision=precision) as e:
            got, st = e.compute_regions(b, with_stats=True)
            _check(b, got, oracle)
            assert st["underflow"] == 0 and st["rescued_cells"] == b.n_cells()
            n = e.stage(b)
            for _ in range(2):
                e.run()
                assert np.array_equal(e.fetch(n), got)


def test_no_allocation_entry_point_on_hopeless_reads(monkeypatch):
    import test_zz_no_alloc as no_alloc
    monkeypatch.setattr(no_alloc, "_batch", lambda: _hopeless(np.random.default_rng(19)))
    no_alloc.test_noalloc_matches_allocating_entry_point()


# reads at the edge of a single strip (253 bases: a unit in FP64 mode; 254: the FP64 list), with some the band takes
def _band_batch():
    rng = np.random.default_rng(23)
    regions = []
    for n in (100, 253, 254, 150, 300):
        hap = W._random_seq(rng, 400)
        reads = [(W._mutate_read(rng, hap, 40, n, 0.01, 0.0, 1, 1), ) for _ in range(3)]
        regions.append(([(r[0], *W._quals(rng, len(r[0]), 10, 40)) for r in reads],
                        [hap, W._substitute(rng, hap, 0.01)]))
    return W._build(regions, "single-strip edge")


@pytest.mark.parametrize("chunks", [0, 2])
def test_fp64_precision_with_the_band_enabled(chunks):
    """Every pair in FP64, whatever the band's options: the values of a context without the band."""
    from biovoltron_b200.pairhmm import PairHMMEngine
    b = _band_batch()
    with PairHMMEngine(precision="f64") as e:
        want = e.compute_regions(b)
    for mode in ("band", "full"):
        with PairHMMEngine(precision="f64", mode=mode, pipeline_chunks=chunks, pipeline_min_pairs=1) as e:
            if mode == "full":
                e.set_band_options(fixed_half=8, margin=2, audit_period=2)
            got, st = e.compute_regions(b, with_stats=True)
            assert np.array_equal(got, want)
            assert st["rescued"] == st["pairs"] == b.n_pairs and st["band_pairs"] == st["band_fallback"] == 0
            n = e.stage(b)
            for _ in range(3):
                e.run()
                assert np.array_equal(e.fetch(n), want)
            d_lo, width, route = e.band_routes()
            assert np.all(route == 3) and not d_lo.any() and not width.any()


def test_labels_and_training_in_an_fp64_context():
    """Band labels and weights do not depend on the context's precision."""
    from biovoltron_b200.pairhmm import PairHMMEngine
    b = _band_batch()
    out = []
    for precision in ("auto", "f64"):
        with PairHMMEngine(precision=precision) as e:
            labels = e.band_labels(b, features=True, extent=True)
            e.band_train(b, epochs=2, batch_size=16)
            out.append([*labels, e.band_weights()])
            scored = e.compute_regions(b)  # the context's precision again
    for x, y in zip(*out):
        assert np.array_equal(x, y)
    assert np.all(out[0][1] > np.iinfo(np.int32).min)
    with PairHMMEngine(precision="f64") as e:
        assert np.array_equal(e.compute_regions(b), scored)


def test_long_read_tuner_keeps_the_choice_per_batch():
    """A sample without long reads changes nothing; a fixed number of warps is in force only if it was the faster; 0
    goes back to the choice per batch.  (The launches of a batch tell the choices apart: clusters of several sizes.)"""
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(29)
    short = W._build([_pair(rng, 150, 300) for _ in range(4)], "short")
    b = W._build([_pair(rng, n, n + 200) for n in (6000, 3000, 1500, 700, 300) for _ in range(4)], "long")
    with PairHMMEngine(precision="f64") as e:
        want, st = e.compute_regions(b, with_stats=True)
        launches = st["kernel_launches"]
        assert e.long_warps() == 4 and not e.long_warps_fixed()
        rep = e.autotune_long(short, repeats=1)
        assert not rep["fixed"] and rep["warps_per_pair"] == e.long_warps() == 4 and not any(rep["fp64_ms"].values())
        got, st = e.compute_regions(b, with_stats=True)
        assert np.array_equal(got, want) and st["kernel_launches"] == launches
        e.set_long_warps(8)
        assert e.long_warps_fixed() and e.compute_regions(b, with_stats=True)[1]["kernel_launches"] != launches
        assert e.autotune_long(short, repeats=1)["fixed"] and e.long_warps() == 8
        rep = e.autotune_long(b, repeats=3)  # clusters are several times faster than any block here
        assert not rep["fixed"] and rep["warps_per_pair"] in (2, 4, 8) and all(rep["fp64_ms"].values())
        assert e.compute_regions(b, with_stats=True)[1]["kernel_launches"] == launches
        e.set_long_warps(2)
        assert e.long_warps_fixed()
        e.set_long_warps(0)
        assert not e.long_warps_fixed() and e.long_warps() == 4
        assert np.array_equal(e.compute_regions(b), want)
