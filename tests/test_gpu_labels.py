"""The label kernel's haplotype-length classes (128 bases each) on either side
of their edges, against the oracle's posterior."""
import numpy as np
import pytest

from biovoltron_b200 import workloads as W
from oracle.oracle import TestcaseArray

pytestmark = pytest.mark.gpu

NONE = np.iinfo(np.int32).min


# haplotypes of 1 base to the longest with a label (1024) and one past it, around multiples of 32 (columns per
# lane) and 128 (classes); reads of one row, longer than the haplotype, and as long as the band takes
@pytest.mark.parametrize("hap_len", [1, 31, 33, 127, 128, 129, 256, 257, 384, 500, 513, 640, 769, 1023, 1024, 1025])
def test_label_classes(oracle, hap_len):
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(hap_len)
    hap = W._random_seq(rng, hap_len)
    haps = [hap, W._substitute(rng, hap, 0.02)]
    reads = []
    for n in (1, 24, 150, 511):
        r = (W._random_seq(rng, n) if n > hap_len else
             W._mutate_read(rng, hap, int(rng.integers(0, hap_len - n + 1)), n, 0.01, 0.01, 1, 3))
        reads.append((r, *W._quals(rng, n, 10, 40)))
    b = W._build([(reads, haps)], "labels")
    tau = 1e-3
    with PairHMMEngine() as e:
        _, lo, hi = e.band_labels(b, tau=tau)
    if hap_len > 1024:
        assert np.all(lo == NONE) and np.all(hi == NONE)
        return
    r, h = b.pair_index()
    tcs = TestcaseArray(b, r, h)
    for k in range(b.n_pairs):
        dmin, pstar = oracle.posterior_diag(tcs, k)
        if pstar is None:
            continue
        # FP32 posteriors against 64 bits: a share within 5 % of tau may fall on either side
        d = np.arange(len(pstar)) + dmin
        strict, loose = d[pstar >= tau * 1.05], d[pstar >= tau * 0.95]
        assert loose.min() <= lo[k] <= strict.min() and strict.max() <= hi[k] <= loose.max(), k


def test_reads_of_a_few_rows(oracle):
    """One to four rows (the backward pass copies rows two ahead), against the oracle's posterior."""
    from biovoltron_b200.pairhmm import PairHMMEngine
    rng = np.random.default_rng(2)
    hap = W._random_seq(rng, 70)
    reads = [(hap[20:20 + n].copy(), *W._quals(rng, n, 20, 40)) for n in (1, 2, 3, 4)]
    b = W._build([(reads, [hap, hap[:40].copy()])], "short reads")
    tau = 1e-3
    with PairHMMEngine() as e:
        _, lo, hi = e.band_labels(b, tau=tau)
    tcs = TestcaseArray(b, *b.pair_index())
    for k in range(b.n_pairs):
        dmin, pstar = oracle.posterior_diag(tcs, k)
        d = np.arange(len(pstar)) + dmin
        strict, loose = d[pstar >= tau * 1.05], d[pstar >= tau * 0.95]
        assert loose.min() <= lo[k] <= strict.min() and strict.max() <= hi[k] <= loose.max(), k
