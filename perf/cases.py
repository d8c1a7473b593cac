"""Performance cases of the PairHMM framework: what is timed, on which inputs, and what it has to give.

A case is one call (or one stage of a program) of the public Python entry
points in ``biovoltron_b200.pairhmm``.  The kinds:

* ``window``   one active region, scored as a haplotype caller scores its
               windows one by one (``PairHMMEngine.compute_regions``, host
               arrays in, log10 matrix out): latency and launches count;
* ``uneven``   a batch of uneven regions (reads 50-250 bp, haplotypes 200-700
               bp, 2-32 haplotypes a region), the shape of the repository's
               ``config1``, host to host;
* ``genome``   regions of a 30x genome (150 bp reads, 2-16 haplotypes of ~450
               bp), the shape of ``config4``: host to host, or the
               device-resident form (staged once, run and fetched each time);
* ``long``     one read of up to 10 kb against one haplotype of up to 12 kb
               per region, ``config2``: the FP32 values underflow and every
               pair takes the FP64 pass;
* ``train``    the band MLP's training on a batch: posterior labels, forward
               and backward passes, Adam, coverage (``band_train``);
* ``genotype`` the device genotyper on a staged, scored batch.

Options met in earnest: precision ``auto`` (FP32 with FP64 rescue) or ``f64``
(every pair, AvxPairHMM's use_double); mode ``full`` or ``band`` (the learned
band); gap qualities as per-base arrays of one value (``arrays``), three
constants for the batch (``uniform``, what SamRecord's constant penalty strings
allow) or per-base arrays that vary (``varied``, as base-quality recalibration
writes them); ``model`` ``avx`` (quality-derived transitions) or ``scalar``
(PairHMM's constant transitions).
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from biovoltron_b200 import workloads as W
from biovoltron_b200.pairhmm import ORIGINAL_DEFAULT, PairHMMEngine

HID, FEAT = 128, 80  # the band MLP's widths


def listed():
    return [
        # a shallow window: few reads, few haplotypes -- the smallest call, all latency
        dict(name="window_20x3", kind="window", reads=20, haps=3, read_len=100, hap_len=220, gaps="uniform",
             model="avx", precision="auto"),
        # the repository's config0: one typical window of a 30-60x sample
        dict(name="window_64x8", kind="window", reads=64, haps=8, read_len=150, hap_len=300, gaps="arrays",
             model="avx", precision="auto"),
        # a caller's queue of a few windows under the scalar model (constant transitions)
        dict(name="uneven_24_scalar", kind="uneven", regions=24, gaps="uniform", model="scalar", precision="auto",
             mode="full"),
        # a small batch of windows with recalibrated (varying) gap qualities
        dict(name="uneven_48_varied", kind="uneven", regions=48, gaps="varied", model="avx", precision="auto",
             mode="full"),
        # an ordinary batch of uneven regions, full DP
        dict(name="uneven_256", kind="uneven", regions=256, gaps="arrays", model="avx", precision="auto",
             mode="full"),
        # the same shapes with every pair in FP64 (use_double)
        dict(name="uneven_64_f64", kind="uneven", regions=64, gaps="arrays", model="avx", precision="f64",
             mode="full"),
        # the same shapes through the learned band, with its rescore
        dict(name="uneven_192_band", kind="uneven", regions=192, gaps="arrays", model="avx", precision="auto",
             mode="band"),
        # a stretch of a 30x genome kept on the device and scored by the full DP
        dict(name="genome_2500_staged", kind="genome", regions=2500, gaps="uniform", mode="full", entry="staged"),
        # the largest: a stretch of a 30x genome, host to host in chunks, through the learned band
        dict(name="genome_8000_band", kind="genome", regions=8000, gaps="uniform", mode="band", entry="call"),
        # long reads: underflow in FP32, scored in FP64
        dict(name="long_40", kind="long", pairs=40, max_read=10000, max_hap=12000),
        # training the band: labels, forward and backward
        dict(name="train_16", kind="train", regions=16, epochs=3, batch=1024),
        # genotyping a scored stretch of genome
        dict(name="genotype_3000", kind="genotype", regions=3000, alleles=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["window", "window", "uneven", "uneven", "uneven", "genome", "genome", "long", "train",
                       "genotype"])
    if kind == "window":
        hap_len = rng.randint(120, 700)
        return dict(kind=kind, reads=_log_int(rng, 1, 300), haps=_log_int(rng, 1, 40),
                    read_len=rng.randint(30, min(250, hap_len)), hap_len=hap_len,
                    gaps=rng.choice(["uniform", "arrays", "varied"]), model=rng.choice(["avx", "avx", "avx", "scalar"]),
                    precision=rng.choice(["auto", "auto", "auto", "f64"]))
    if kind == "uneven":
        form = rng.choice(["full", "full", "band", "f64", "scalar"])
        top = {"full": 256, "band": 192, "f64": 64, "scalar": 64}[form]
        return dict(kind=kind, regions=_log_int(rng, 3, top), gaps=rng.choice(["uniform", "arrays", "varied"]),
                    model="scalar" if form == "scalar" else "avx", precision="f64" if form == "f64" else "auto",
                    mode="band" if form == "band" else "full")
    if kind == "genome":
        mode = rng.choice(["full", "band"])
        return dict(kind=kind, regions=_log_int(rng, 60, 8000 if mode == "band" else 2500),
                    gaps=rng.choice(["uniform", "arrays"]), mode=mode, entry=rng.choice(["staged", "call"]))
    if kind == "long":
        return dict(kind=kind, pairs=_log_int(rng, 2, 40), max_read=_log_int(rng, 300, 10000),
                    max_hap=rng.randint(1000, 12000))
    if kind == "train":
        return dict(kind=kind, regions=rng.randint(3, 16), epochs=rng.randint(1, 3),
                    batch=rng.choice([256, 500, 1024, 2048]))
    return dict(kind=kind, regions=_log_int(rng, 50, 3000), alleles=rng.randint(2, 4))


# --- inputs ---------------------------------------------------------------------
def _window(c, rng):
    """One region: haplotypes differ from a base sequence by 1 % SNVs and up to
    two indels of 1-10 bp, reads come from them with 1 % substitutions, base
    qualities 10-40 (the model of the repository's config0)."""
    acgt = np.frombuffer(b"ACGT", np.uint8)

    def snv(s):
        hit = rng.random(s.size) < 0.01
        return np.where(hit, acgt[rng.integers(0, 4, s.size)], s)

    base = acgt[rng.integers(0, 4, c["hap_len"])]
    haps = []
    for _ in range(c["haps"]):
        h = snv(base)
        for _ in range(int(rng.integers(0, 3))):
            n = int(rng.integers(1, 11))
            at = int(rng.integers(1, h.size - n - 1))
            h = np.concatenate([h[:at], acgt[rng.integers(0, 4, n)], h[at:]] if rng.random() < 0.5
                               else [h[:at], h[at + n:]])
        haps.append(h)
    reads = []
    for _ in range(c["reads"]):
        src = haps[int(rng.integers(0, len(haps)))]
        n = min(c["read_len"], src.size)
        at = int(rng.integers(0, src.size - n + 1))
        reads.append(snv(src[at:at + n]))
    off = lambda parts: np.concatenate([[0], np.cumsum([p.size for p in parts])]).astype(np.int64)  # noqa: E731
    rb = np.concatenate(reads)
    one = lambda v: np.full(rb.size, v, np.uint8)  # noqa: E731
    return W.RegionBatch(read_bases=rb, read_q=rng.integers(10, 41, rb.size).astype(np.uint8), read_i=one(45),
                         read_d=one(45), read_c=one(10), read_offsets=off(reads), hap_bases=np.concatenate(haps),
                         hap_offsets=off(haps), region_reads=np.array([0, len(reads)], np.int64),
                         region_haps=np.array([0, len(haps)], np.int64), name="window")


@functools.lru_cache(maxsize=4)
def _template(kind, size, max_read, max_hap):
    """The repository's workload of that shape: it fixes the counts and lengths of a case."""
    if kind == "long":
        return W.config2(seed=size, n_pairs=size, max_read=max_read, max_hap=max_hap)
    return (W.config1 if kind in ("uneven", "train") else W.config4)(seed=size, n_regions=size)


def _shape(case):
    return _template(case["kind"], case.get("regions") or case["pairs"], case.get("max_read"), case.get("max_hap"))


def _inputs(case, seed):
    """The case's batch and the constants passed instead of its gap arrays.
    Counts and lengths belong to the case, the contents to the seed: every
    region's bases under a permutation of its own, new base qualities, and a
    few more substitutions in the reads."""
    rng = np.random.default_rng([seed, 77])
    if case["kind"] == "window":
        b = _window(case, rng)
    else:
        t = _shape(case)
        order = rng.permuted(np.tile(np.arange(4, dtype=np.uint8), (t.n_regions, 1)), axis=1).ravel()
        code = np.zeros(256, np.int32)
        code[list(b"ACGT")] = range(4)
        acgt = np.frombuffer(b"ACGT", np.uint8)

        def bases(flat, offsets, owner):
            region = np.repeat(np.repeat(np.arange(t.n_regions, dtype=np.int32), np.diff(owner)), np.diff(offsets))
            return order[4 * region + code[flat]]

        rb = bases(t.read_bases, t.read_offsets, t.region_reads)
        hit = rng.integers(0, rb.size, rb.size // 500)
        rb[hit] = rng.integers(0, 4, hit.size, dtype=np.uint8)
        lo, hi = (5, 30) if case["kind"] == "long" else (10, 40)
        b = dataclasses.replace(t, read_bases=acgt[rb],
                                hap_bases=acgt[bases(t.hap_bases, t.hap_offsets, t.region_haps)],
                                read_q=rng.integers(lo, hi + 1, rb.size, dtype=np.uint8))
    gaps = case.get("gaps", "arrays")
    if gaps == "varied":
        b.read_i = rng.integers(30, 50, b.read_bases.size, dtype=np.uint8)
        b.read_d = rng.integers(30, 50, b.read_bases.size, dtype=np.uint8)
        b.read_c = rng.integers(8, 14, b.read_bases.size, dtype=np.uint8)
    uniform = None
    if gaps == "uniform":
        uniform = (0, 0, 0) if case.get("model") == "scalar" else (45, 45, 10)
    return b, uniform


def _pinned(a):
    """A page-locked copy (what a program that streams batches keeps its arrays in)."""
    t = torch.empty(max(a.size, 1), dtype=torch.from_numpy(a[:0]).dtype, pin_memory=torch.cuda.is_available())
    out = t.numpy()[:a.size]
    out[:] = a
    return out


def band_weights(seed=5):
    """Band MLP parameters whose outputs behave like a trained network's: a few
    diagonals around the seed, wider with uncovered read ends and mismatching
    ends.  (Training them is the ``train`` case; these need no batch.)  Six
    hidden units carry the features that matter, the others small noise."""
    rng = np.random.default_rng(seed)
    w1 = (rng.standard_normal((HID, FEAT)) * 0.01).astype(np.float32)
    w2 = (rng.standard_normal((HID, HID)) * 0.01).astype(np.float32)
    w3 = (rng.standard_normal((2, HID)) * 0.01).astype(np.float32)
    b1, b2 = np.zeros(HID, np.float32), np.zeros(HID, np.float32)
    # features 72, 73: uncovered read ends / 32; 76, 77: mismatches of the read ends / 16; 65: hits off the window
    for unit, feat in enumerate((72, 73, 76, 77, 65)):
        w1[unit] = 0
        w1[unit, feat] = 1
        w2[unit] = 0
        w2[unit, unit] = 1
    w3[0, :5] = (-3, -5, -3, -5, -8)
    w3[1, :5] = (5, 3, 5, 3, 8)
    b3 = np.array([-0.8, 0.8], np.float32)
    return np.concatenate([x.ravel() for x in (w1, b1, w2, b2, w3, b3)])


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case = case
    b, s.gaps = _inputs(case, seed)
    s.eng = PairHMMEngine(precision=case.get("precision", "auto"))
    if case.get("mode") == "band":
        s.eng.set_band_weights(band_weights())
        s.eng.set_band_options(enabled=True, use_mlp=True)
    if case.get("model") == "scalar":
        s.eng.set_transitions(ORIGINAL_DEFAULT)
    if case["kind"] == "genome":  # large batches: page-locked inputs and results
        for f in ("read_bases", "read_q", "read_offsets", "hap_bases", "hap_offsets") + (
                () if s.gaps else ("read_i", "read_d", "read_c")):
            setattr(b, f, _pinned(getattr(b, f)))
    s.batch = b
    s.out = _pinned(np.zeros(b.n_pairs)) if case["kind"] == "genome" else np.zeros(b.n_pairs)
    if case.get("entry") == "staged" or case["kind"] == "genotype":
        s.n = s.eng.stage(b, uniform_gaps=s.gaps)
        s.eng.run()
    if case["kind"] == "genotype":
        rng = np.random.default_rng([seed, 78])
        a = case["alleles"]
        s.alleles = np.full(b.n_regions, a, np.int32)
        s.hap_allele = rng.integers(0, a, b.n_haps).astype(np.int32)
        s.overlaps = (rng.random(b.n_reads) < 0.9).astype(np.uint8)
        nr = np.diff(b.region_reads)
        s.region_of = np.repeat(np.arange(b.n_regions), nr)
        s.place = np.arange(b.n_reads) - np.repeat(b.region_reads[:-1], nr)
    return s


def run(s):
    kind = s.case["kind"]
    if kind == "train":
        rep = s.eng.band_train(s.batch, epochs=s.case["epochs"], batch_size=s.case["batch"])
        return {"weights": s.eng.band_weights(), "loss": np.array([rep["first_loss"], rep["last_loss"]], np.float32),
                "counts": [rep["pairs"], rep["labelled"], rep["steps"]],
                "fractions": [rep["cover_frac"], rep["band_frac"]]}
    if kind == "genotype":
        g = s.eng.genotype_staged(s.batch, s.alleles, s.hap_allele, s.overlaps)
        past = s.place >= g["kept_count"][s.region_of]  # slots past a region's kept reads are not written
        g["kept_reads"][past] = -1
        g["allele_lik"].reshape(-1, s.case["alleles"])[past] = 0
        return {k: g[k] for k in ("kept_count", "kept_reads", "allele_lik", "genotype_lik")}
    if s.case.get("entry") == "staged":
        s.eng.run()
        return s.eng.fetch(s.n, out=s.out)
    return s.eng.compute_regions(s.batch, out=s.out, uniform_gaps=s.gaps)


# --- what a pass cannot do without -------------------------------------------------
def _sizes(case):
    """(reads, haplotypes, pairs, read bases, haplotype bases, cells) of a case's batch."""
    if case["kind"] == "window":
        r, h, rl, hl = case["reads"], case["haps"], case["read_len"], case["hap_len"]
        return r, h, r * h, r * rl, h * hl, r * h * rl * hl
    t = _shape(case)
    nr, nh = np.add.reduceat(t.read_lengths(), t.region_reads[:-1]), np.add.reduceat(t.hap_lengths(), t.region_haps[:-1])
    return t.n_reads, t.n_haps, t.n_pairs, int(nr.sum()), int(nh.sum()), int((nr * nh).sum())


def work(case):
    r, h, p, rb, hb, cells = _sizes(case)
    per_base = 2 if case.get("gaps") == "uniform" else 5
    io = rb * per_base + hb + 8 * (r + h) + 8 * p
    if case["kind"] == "genotype":
        a = case["alleles"]
        return {"bytes": 8 * p + 8 * r * a + 5 * r + 4 * h + 4 * a * (a + 1) * case["regions"], "flops": 2 * p}
    if case["kind"] == "train":
        mlp = 2 * (FEAT * HID + HID * HID + 2 * HID)
        return {"bytes": io, "flops": 32 * cells + 3 * mlp * p * case["epochs"]}
    if case.get("mode") == "band":  # 12 flops per cell of a band of 16 diagonals, and the MLP
        return {"bytes": io, "flops": 12 * 16 * p * (rb / r) + 2 * (FEAT * HID + HID * HID + 2 * HID) * p}
    return {"bytes": io, "flops": 12 * cells}


# --- the values in 64 bits ------------------------------------------------------------
MOST_CELLS = 1.7e11  # beyond it the 64-bit pass below takes too long


def exact(case, seed):
    if case["kind"] in ("train", "genotype") or _sizes(case)[5] > MOST_CELLS:
        return None
    b, _ = _inputs(case, seed)
    return _log10_likelihoods(b, ORIGINAL_DEFAULT if case.get("model") == "scalar" else None)


def _rows(b, reads, n, trans, dev):
    """Per pair and read row (row 0 = the initial row): base codes and the row's probabilities."""
    at = torch.from_numpy(b.read_offsets[:-1].astype(np.int64)).to(dev)[reads]
    ln = torch.from_numpy(np.diff(b.read_offsets).astype(np.int64)).to(dev)[reads]
    j = torch.arange(-1, n, device=dev)[None, :]
    ok = (j >= 0) & (j < ln[:, None])
    ix = torch.where(ok, at[:, None] + j, torch.zeros_like(at[:, None]))
    code = torch.zeros(256, dtype=torch.uint8)
    for k, ch in enumerate(b"ACTGN"):
        code[ch] = k
    phred = torch.pow(torch.tensor(10.0, dtype=torch.float64), -torch.arange(128, dtype=torch.float64) / 10).to(dev)
    take = lambda a: torch.from_numpy(a).to(dev)[ix].long()  # noqa: E731
    prob = lambda a: torch.where(ok, phred[take(a) & 127], torch.zeros((), dtype=torch.float64, device=dev))  # noqa: E731
    eps = prob(b.read_q)
    p = {"code": torch.where(ok, code.to(dev)[take(b.read_bases)], torch.full_like(ix, 6, dtype=torch.uint8)),
         "hit": torch.where(ok, 1 - eps, torch.zeros_like(eps)), "miss": eps / 3}
    if trans is None:
        i, d, g = prob(b.read_i), prob(b.read_d), prob(b.read_c)
        p |= {"mm": 1 - (i + d), "mx": i, "my": d, "xx": g, "yy": g, "xm": 1 - g, "ym": 1 - g}
    else:
        p |= dict(zip(("mm", "mx", "my", "xm", "xx", "ym", "yy"), trans))
    return p, ln


def _log10_likelihoods(b, trans):
    """log10 of every pair's forward likelihood, region by region, read-major:
    the Match/Insert/Delete recurrence on whole anti-diagonals, many pairs at a
    time.  Long reads carry a power of two per row."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    reads, haps = b.pair_index()
    rl, hl = b.read_lengths()[reads], b.hap_lengths()[haps]
    out = torch.zeros(len(reads), dtype=torch.float64, device=dev)
    order = np.lexsort((hl, rl))
    k = 0
    while k < len(order):
        # the next pairs in order of length, as many as 12 million rows hold
        n = max(1, min(len(order) - k, int(12e6 // (rl[order[min(len(order) - 1, k + 20000)]] + 1))))
        pick = order[k:k + n]
        k += n
        out[torch.from_numpy(pick).to(dev)] = _group(b, torch.from_numpy(reads[pick]).to(dev), haps[pick], trans, dev)
    return out.cpu().numpy()


def _group(b, reads, haps, trans, dev):
    n = int(b.read_lengths()[reads.cpu().numpy()].max())
    p, ln = _rows(b, reads, n, trans, dev)
    hl = torch.from_numpy(b.hap_lengths()[haps]).to(dev)
    h = int(hl.max())
    # haplotype codes reversed, so that an anti-diagonal's columns are one slice (5: outside)
    code = torch.full((256,), 0, dtype=torch.uint8)
    for v, ch in enumerate(b"ACTGN"):
        code[ch] = v
    start = torch.from_numpy(b.hap_offsets[:-1].astype(np.int64)[haps]).to(dev)
    col = torch.arange(h + n, -n - 1, -1, device=dev)[None, :] - 1  # 0-based column of each slot
    ok = (col >= 0) & (col < hl[:, None])
    hr = torch.where(ok, code.to(dev)[torch.from_numpy(b.hap_bases).to(dev)[torch.where(
        ok, start[:, None] + col, torch.zeros_like(start[:, None]))].long()],
        torch.full((), 5, dtype=torch.uint8, device=dev))
    P, scaled = len(haps), n > 400
    z = lambda: torch.zeros(P, n + 1, dtype=torch.float64, device=dev)  # noqa: E731
    m1, x1, y1, m2, x2, y2 = z(), z(), z(), z(), z(), z()
    init = 2.0 ** (0 if scaled else 1000)
    start_y = init / hl.double()
    y1[:, 0] = start_y
    y2[:, 0] = start_y  # row 0 holds it in every column; only columns >= 0 are read
    expo, factor = z(), None  # true values are stored * 2^expo; factor: row r-1's scale in row r's
    total = torch.full((P,), -math.inf, dtype=torch.float64, device=dev)
    last = ln[:, None]
    any_n = (p["code"] == 4)
    for t in range(2, n + h + 1):
        hs = hr[:, h + n - t:h + 2 * n - t + 1]  # row r: column t - r
        e = torch.where((hs == p["code"]) | any_n | (hs == 4), p["hit"], p["miss"])
        e = torch.where(hs == 5, torch.zeros_like(e), e)[:, 1:]
        row = lambda name: p[name][:, 1:] if isinstance(p[name], torch.Tensor) else p[name]  # noqa: E731
        m = (row("mm") * m2[:, :-1] + row("xm") * x2[:, :-1] + row("ym") * y2[:, :-1]) * e
        x = row("mx") * m1[:, :-1] + row("xx") * x1[:, :-1]
        if factor is not None:
            m, x = m * factor, x * factor
        y = row("my") * m1[:, 1:] + row("yy") * y1[:, 1:]
        m2, x2, y2 = m1, x1, y1
        m1, x1, y1 = z(), z(), z()
        m1[:, 1:], x1[:, 1:], y1[:, 1:] = m, x, y
        y1[:, 0] = y2[:, 0]
        s = (m1 + x1).gather(1, last)[:, 0]
        c = t - ln
        s = torch.where((c >= 1) & (c <= hl), s, torch.zeros_like(s))
        total = torch.logaddexp2(total, torch.log2(s) + expo.gather(1, last)[:, 0])
        if scaled and t % 32 == 0:
            top = torch.stack([m1, x1, y1, m2, x2, y2]).amax(0)
            shift = torch.where(top > 0, torch.floor(torch.log2(top)), torch.zeros_like(top))
            half = torch.floor(shift / 2)  # in two factors: 2^-shift may lie outside the range
            for v in (m1, x1, y1, m2, x2, y2):
                v.mul_(torch.exp2(-half)).mul_(torch.exp2(half - shift))
            expo = expo + shift
            # rows that nothing has reached yet take the scale of the last row that has a value
            reach = torch.where(top > 0, torch.arange(n + 1, device=dev)[None, :], -1).cummax(1).values
            expo = expo.gather(1, reach)
            factor = torch.exp2((expo[:, :-1] - expo[:, 1:]).clamp(-1000, 1000))
    return (total - (0 if scaled else 1000)) * math.log10(2)
