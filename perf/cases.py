"""The work that users of this library have it do, as measurable cases.

Each case is one call (or the short loop) that a population-genetics script
makes with its data already in hand: an int8 haplotype or dosage matrix and
its positions on the GPU.  ``listed()`` holds twelve of them, ``draw(rng)``
gives more of the same kinds and ranges, ``run(state)`` makes one pass through
the public entry points and ``exact(case, seed)`` evaluates the same estimators
in 64 bits with plain torch.

Panels come from the copying model of this repository's tests and benchmark
(founders with Beta(0.3, 0.3) allele frequencies, founder switches, allele
flips, entries missing completely at random), about one SNP per 100 bp.
"""
import itertools
import math

import numpy as np
import torch

from pg_gpu_gb300 import ld_pipeline, ld_statistics, moments_ld
from pg_gpu_gb300.genotype_matrix import GenotypeMatrix
from pg_gpu_gb300.haplotype_matrix import HaplotypeMatrix

SPACING = 100  # base pairs per SNP on average


def listed():
    return [
        # moments two-population LD of a chromosome arm: the headline size
        dict(name="two_pops_arm", kind="two_pops", n=1000, snps=200_000, max_kb=1000, bins=20,
             missing=0.02, raw=True),
        # one population, a small region: launch latency and host work count
        dict(name="one_pop_region", kind="one_pop", n=200, snps=2000, max_kb=100, bins=20,
             missing=0.0, raw=False),
        # moments_ld with three populations (haplotypes), the out-of-Africa set-up
        dict(name="moments_hap_3", kind="moments_hap", pops=3, n=200, snps=50_000, max_kb=100,
             bins=12, missing=0.02),
        # moments_ld on unphased genotypes with its default two populations
        dict(name="moments_geno_2", kind="moments_geno", pops=2, n=500, snps=100_000, max_kb=100,
             bins=12, missing=0.03),
        # every pair of a distance band: counts, n, r^2, DD, Dz and pi2 per pair
        dict(name="hap_band", kind="hap_band", n=2000, snps=100_000, max_kb=100, missing=0.02),
        # the same on unphased genotypes, every output
        dict(name="geno_band", kind="geno_band", n=1000, snps=100_000, max_kb=100, missing=0.03),
        # Kelly's ZnS over uneven windows of a genome, one call
        dict(name="windowed_zns", kind="zns", n=400, windows=512, lo=500, hi=20_000, missing=0.0),
        # Kim and Nielsen's omega in a sweep scan's windows, from r^2 (the ratio
        # of sigma_D^2 means has no stable value where their sum crosses zero)
        dict(name="windowed_omega", kind="omega", n=401, windows=200, lo=200, hi=2000,
             missing=0.01),
        # a script's own loop over pair chunks: counts of two populations and the
        # 15 statistics of each chunk
        dict(name="pair_chunks", kind="chunks", n=100, snps=4000, max_kb=20, chunk=250_000,
             missing=0.02),
        # Rogers-Huff r of all variant pairs of a region (scikit-allel's use)
        dict(name="rogers_huff", kind="rogers_huff", n=1000, snps=3000, missing=0.0),
        # r^2 decay: percentiles of r^2 by distance over all pairs of a region
        dict(name="r2_decay", kind="r2_decay", n=300, snps=5001, bins=15, missing=0.02),
        # all pairs of a small region: joint counts, then four statistics of them
        dict(name="all_pairs", kind="all_pairs", n=200, snps=2000, missing=0.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any kind, sizes spread over its range (odd ones among them)."""
    kind = rng.choice([c["kind"] for c in listed()])
    c = dict(kind=kind, missing=rng.choice([0.0, 0.01, 0.02, 0.03]))
    if kind == "two_pops":
        c.update(n=_log_int(rng, 40, 1000), snps=_log_int(rng, 20_000, 200_000),
                 max_kb=rng.choice([100, 300, 1000]), bins=rng.randint(8, 24),
                 raw=rng.choice([True, False]))
    elif kind == "one_pop":
        c.update(n=_log_int(rng, 30, 2000), snps=_log_int(rng, 1500, 20_000), max_kb=100,
                 bins=rng.randint(4, 20), raw=rng.choice([True, False]))
    elif kind == "moments_hap":
        pops = rng.choice([2, 3, 3, 4])
        c.update(pops=pops, n=_log_int(rng, 30, 400), snps=_log_int(rng, 10_000, 50_000),
                 max_kb=100, bins=rng.randint(6, 14))
    elif kind == "moments_geno":
        pops = rng.choice([1, 2, 2, 3, 4])
        c.update(pops=pops, n=_log_int(rng, 30, 500),
                 snps=_log_int(rng, 10_000, 100_000 if pops < 3 else 30_000), max_kb=100,
                 bins=rng.randint(6, 14))
    elif kind in ("hap_band", "geno_band"):
        c.update(n=_log_int(rng, 50, 2000 if kind == "hap_band" else 1000),
                 snps=_log_int(rng, 5000, 100_000), max_kb=rng.choice([10, 30, 100]))
    elif kind == "zns":
        c.update(n=_log_int(rng, 50, 500), windows=rng.randint(20, 512), lo=200,
                 hi=_log_int(rng, 1000, 20_000))
    elif kind == "omega":
        c.update(n=_log_int(rng, 50, 500), windows=rng.randint(20, 200), lo=100,
                 hi=_log_int(rng, 400, 2000))
    elif kind == "chunks":
        c.update(n=_log_int(rng, 30, 300), snps=_log_int(rng, 1500, 5000),
                 max_kb=rng.choice([10, 20]), chunk=rng.choice([200_000, 500_000, 1_000_000]))
    elif kind == "rogers_huff":
        c.update(n=_log_int(rng, 50, 1000), snps=_log_int(rng, 500, 3000), missing=0.0)
    elif kind == "r2_decay":
        c.update(n=_log_int(rng, 50, 500), snps=_log_int(rng, 500, 5001), bins=rng.randint(5, 20))
    else:
        c.update(n=_log_int(rng, 50, 500), snps=_log_int(rng, 300, 2000))
    return c


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _positions(snps, seed):
    """Sorted distinct int64 positions on the GPU, SPACING apart on average."""
    u = np.random.default_rng(seed).random(snps)
    gaps = 1 + np.floor(-np.log1p(-u) * (SPACING - 1))
    return torch.as_tensor(np.cumsum(gaps.astype(np.int64)), device="cuda")


def _panel(seed, pops, n, snps, missing):
    """int8 (pops * n, snps) haplotypes and their positions, on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rng = np.random.default_rng(seed)
    founders, switch, flip, pop_flip = 40, 1e-3, 1e-3, 0.1

    def rand(*shape):
        return torch.rand(shape, generator=g, device="cuda")

    p = torch.as_tensor(rng.beta(0.3, 0.3, snps), dtype=torch.float32, device="cuda")
    pool = (rand(founders, snps) < p).to(torch.int8)
    hap = torch.empty((pops * n, snps), dtype=torch.int8, device="cuda")
    for k in range(pops):
        mine = pool ^ (rand(founders, snps) < pop_flip).to(torch.int8) if pops > 1 else pool
        step = max(1, (1 << 27) // snps)  # haplotypes at a time
        for r in range(0, n, step):
            m = min(step, n - r)
            seg = torch.cumsum(rand(m, snps) < switch, 1, dtype=torch.int32)
            choice = torch.randint(0, founders, (m, int(seg.max()) + 1), generator=g,
                                   device="cuda")
            h = torch.gather(mine, 0, torch.gather(choice, 1, seg.long()))
            h ^= (rand(m, snps) < flip).to(torch.int8)
            if missing:
                h[rand(m, snps) < missing] = -1
            hap[k * n + r:k * n + r + m] = h
    return hap, _positions(snps, seed)


def _dosages(seed, pops, n, snps, missing):
    hap, pos = _panel(seed, pops, 2 * n, snps, 0.0)
    geno = hap[0::2] + hap[1::2]
    if missing:
        g = torch.Generator(device="cuda")
        g.manual_seed(seed + 1)
        for r in range(0, geno.shape[0], 100):
            part = geno[r:r + 100]
            part[torch.rand(part.shape, generator=g, device="cuda") < missing] = -1
    return geno, pos


def _sets(pops, n):
    return {f"pop{k}": list(range(k * n, (k + 1) * n)) for k in range(pops)}


def _windows(case, seed):
    """Starts and stops of consecutive SNP windows of log-uniform size."""
    rng = np.random.default_rng(seed + 2)
    size = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), case["windows"]))
    stop = np.cumsum(size.astype(np.int64))
    return np.concatenate([[0], stop[:-1]]), stop


def _bins(case):
    if case["kind"] == "r2_decay":
        return np.linspace(0, case["snps"] * SPACING, case["bins"] + 1)
    return np.logspace(3, 3 + math.log10(case["max_kb"]), case["bins"] + 1)


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    s = dict(case=case)
    if kind in ("zns", "omega"):
        s["start"], s["stop"] = _windows(case, seed)
        s["hap"], s["pos"] = _panel(seed, 1, n, int(s["stop"][-1]), case["missing"])
    elif kind in ("moments_geno", "geno_band", "rogers_huff"):
        pops = case.get("pops", 1)
        s["geno"], s["pos"] = _dosages(seed, pops, n, case["snps"], case["missing"])
        s["sets"] = _sets(pops, n)
    else:
        pops = 2 if kind in ("two_pops", "chunks") else case.get("pops", 1)
        s["hap"], s["pos"] = _panel(seed, pops, n, case["snps"], case["missing"])
        s["sets"] = _sets(pops, n)
    if kind in ("hap_band", "geno_band", "chunks"):
        # one site map for every data set: the outputs have one entry per pair in reach
        s["pos"] = _positions(case["snps"], case["snps"])
    if "bins" in case:
        s["bins"] = _bins(case)
    return s


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "two_pops":
        hm = HaplotypeMatrix(s["hap"], s["pos"], sample_sets=s["sets"])
        out = hm.compute_ld_statistics_gpu_two_pops(s["bins"], "pop0", "pop1", raw=case["raw"])
        return np.array([list(v.values()) for v in out.values()])
    if kind == "one_pop":
        hm = HaplotypeMatrix(s["hap"], s["pos"])
        out = hm.compute_ld_statistics_gpu_single_pop(s["bins"], raw=case["raw"])
        return np.array(list(out.values()))
    if kind == "moments_hap":
        hm = HaplotypeMatrix(s["hap"], s["pos"], sample_sets=s["sets"])
        return moments_ld.compute_ld_statistics(haplotype_matrix=hm, pops=list(s["sets"]),
                                                bp_bins=s["bins"], report=False)["sums"]
    if kind == "moments_geno":
        gm = GenotypeMatrix(s["geno"], s["pos"], sample_sets=s["sets"])
        return moments_ld.compute_ld_statistics(genotype_matrix=gm, pops=list(s["sets"]),
                                                bp_bins=s["bins"], use_genotypes=True,
                                                report=False)["sums"]
    if kind == "hap_band":
        return ld_pipeline.pairs_within_distance_statistics(s["hap"], s["pos"],
                                                            case["max_kb"] * 1000)
    if kind == "geno_band":
        return ld_pipeline.genotype_pairs_within_distance_statistics(s["geno"], s["pos"],
                                                                     case["max_kb"] * 1000)
    if kind == "zns":
        return ld_statistics.windowed_zns(HaplotypeMatrix(s["hap"], s["pos"]), s["start"],
                                          s["stop"])
    if kind == "omega":
        return ld_statistics.windowed_omega(HaplotypeMatrix(s["hap"], s["pos"]), s["start"],
                                            s["stop"], estimator="r2")
    if kind == "chunks":
        out = []
        for i, j in ld_pipeline.iter_pairs_within_distance(s["pos"], case["max_kb"] * 1000,
                                                           case["chunk"]):
            c, v = zip(*(ld_pipeline.compute_counts_for_pairs(s["hap"], i, j, rows)
                         for rows in s["sets"].values()))
            stats = ld_pipeline.compute_two_pop_statistics_batch(c[0], c[1], v[0], v[1])
            out.append((i, j, *c, stats))
        return out
    if kind == "rogers_huff":
        return ld_statistics.rogers_huff_r(GenotypeMatrix(s["geno"], s["pos"]))
    if kind == "r2_decay":
        hm = HaplotypeMatrix(s["hap"], s["pos"])
        return hm.windowed_r_squared(s["bins"], percentile=[50, 90])
    hm = HaplotypeMatrix(s["hap"], s["pos"])
    counts, n_valid = hm.tally_gpu_haplotypes()
    stats = ld_statistics.compute_ld_statistics(counts, ["dd", "dz", "pi2", "r_squared"],
                                                n_valid=n_valid)
    return counts, n_valid, stats


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _band_pairs(case):
    w = case["max_kb"] * 1000 / SPACING
    return case["snps"] * w - w * w / 2 if w < case["snps"] else case["snps"] ** 2 / 2


def work(case):
    kind, n = case["kind"], case["n"]
    if kind in ("zns", "omega"):
        lo, hi, k = case["lo"], case["hi"], math.log(case["hi"] / case["lo"])
        snps = case["windows"] * (hi - lo) / k
        pairs = case["windows"] * (hi * hi - lo * lo) / (4 * k)
        return {"bytes": n * snps + 24 * case["windows"], "flops": 8 * n * pairs}
    pops = 2 if kind in ("two_pops", "chunks") else case.get("pops", 1)
    rows, snps = pops * n, case["snps"]
    pairs = snps * (snps - 1) / 2 if "max_kb" not in case else _band_pairs(case)
    per_pair = {"hap_band": 36, "geno_band": 56, "chunks": 8 + 32 + 120, "rogers_huff": 8,
                "all_pairs": 16 + 32}.get(kind, 0)
    geno = kind in ("moments_geno", "geno_band", "rogers_huff")
    return {"bytes": rows * snps + 8 * snps + per_pair * pairs,
            "flops": (18 if geno else 8) * rows * pairs}


# --------------------------------------------------------------------------
# the same estimators in 64 bits
#
# Every statistic is a product of linear forms of the pair's class frequencies
# (haplotypes 11, 10, 01, 00 or dosages 00 .. 22), one population each; a
# population's product of k forms is estimated without bias by averaging over
# k distinct individuals: the inclusion-exclusion sum over set partitions
# below, divided by n (n - 1) ... (n - k + 1).
# --------------------------------------------------------------------------
_HAP = {"11": (1, 0, 0, 0), "10": (0, 1, 0, 0), "01": (0, 0, 1, 0), "00": (0, 0, 0, 1),
        "p": (1, 1, 0, 0), "P": (0, 0, 1, 1), "q": (1, 0, 1, 0), "Q": (0, 1, 0, 1),
        "a": (-1, -1, 1, 1), "b": (-1, 1, -1, 1)}
_AB = [(a / 2, b / 2) for a in range(3) for b in range(3)]
_GENO = {"11": [a * b for a, b in _AB], "10": [a * (1 - b) for a, b in _AB],
         "01": [(1 - a) * b for a, b in _AB], "00": [(1 - a) * (1 - b) for a, b in _AB],
         "p": [a for a, _ in _AB], "P": [1 - a for a, _ in _AB],
         "q": [b for _, b in _AB], "Q": [1 - b for _, b in _AB],
         "a": [1 - 2 * a for a, _ in _AB], "b": [1 - 2 * b for _, b in _AB]}


def _partitions(k):
    if k == 0:
        return [[]]
    out = []
    for part in _partitions(k - 1):
        out.append(part + [[k - 1]])
        out += [part[:x] + [part[x] + [k - 1]] + part[x + 1:] for x in range(len(part))]
    return out


_PART = {k: _partitions(k) for k in range(1, 5)}


class _Pop:
    """Class counts (classes, N) of one population for N pairs."""

    def __init__(self, c, forms):
        self.c, self.forms, self.n, self.seen = c, forms, c.sum(0), {}

    def form(self, names):
        coef = [math.prod(v) for v in zip(*(self.forms[x] for x in names))]
        key = tuple(coef)
        if key not in self.seen:
            t = None
            for w, c in zip(coef, self.c):
                if w:
                    t = c * w if t is None else t.add_(c, alpha=w)
            self.seen[key] = t
        return self.seen[key]

    def draws(self, names):
        names = tuple(sorted(names))
        if names not in self.seen:
            tot = torch.zeros_like(self.n)
            for part in _PART[len(names)]:
                fs = [self.form([names[x] for x in block]) for block in part]
                if any(f is None for f in fs):
                    continue
                w = math.prod((-1) ** (len(b) - 1) * math.factorial(len(b) - 1) for b in part)
                t = fs[0] * w
                for f in fs[1:]:
                    t *= f
                tot += t
            self.seen[names] = tot
        return self.seen[names]

    def falling(self, k):
        key = ("n", k)
        if key not in self.seen:
            d = self.n.clone()
            for x in range(1, k):
                d *= self.n - x
            self.seen[key] = d
        return self.seen[key]


def _mean(pops, terms):
    """Sum of weight x the product over populations of their estimates; a term
    is (weight, [(population, form), ...])."""
    out = 0
    for w, fs in terms:
        by = {}
        for p, f in fs:
            by.setdefault(p, []).append(f)
        t = None
        for p, names in by.items():
            d = pops[p].falling(len(names))
            v = torch.where(d > 0, pops[p].draws(names) / d.clamp(min=1), torch.zeros_like(d))
            t = v if t is None else t * v
        out = out + w * t
    return out


def _times(x, y):
    return [(v * w, f + g) for v, f in x for w, g in y]


def _statistics(P, geno):
    """(weight, forms) terms of the moments statistics of P populations, in moments' order."""
    scale = 2.0 if geno else 1.0

    def D(i):
        return [(scale, [(i, "11"), (i, "00")]), (-scale, [(i, "10"), (i, "01")])]

    stats = [_times(D(i), D(j)) for i in range(P) for j in range(i, P)]
    for i in range(P):
        for j in range(P):
            for k in range(j, P):
                two = _times(D(i), [(0.5, [(j, "a"), (k, "b")])])
                stats.append(two + _times(D(i), [(0.5, [(k, "a"), (j, "b")])]))
    for i in range(P):
        for j in range(i, P):
            for k in range(i, P):
                for l in range(k, P):
                    if (k == i == l and j != i) or (i == k and l < j):
                        continue
                    orders = {(*x, *y) for u, v in (((i, j), (k, l)), ((k, l), (i, j)))
                              for x in (u, u[::-1]) for y in (v, v[::-1])}
                    count = max([i, j, k, l].count(x) for x in (i, j, k, l))
                    if count == 3 and not geno:
                        # the haplotype form of three draws from one population
                        # takes two of them at the first SNP
                        orders = {o for o in orders if o[0] == o[1]}
                    stats.append([(1 / len(orders), [(a, "p"), (b, "P"), (c, "q"), (d, "Q")])
                                  for a, b, c, d in sorted(orders)])
    return stats


def _planes(x, classes):
    return torch.stack([(x == v).to(torch.float32) for v in classes])


def _row_blocks(pos, max_dist, most):
    """(i0, i1, j1): rows i0..i1 and the columns i0..j1 they pair with."""
    m = len(pos)
    end = np.searchsorted(pos, pos + max_dist, side="right")
    i0 = 0
    while i0 < m - 1:
        i1 = i0 + 1
        while i1 < m and (i1 + 1 - i0) * (end[i1] - i0) <= most:
            i1 = min(m, i1 + max(1, (i1 - i0) // 8))
        yield i0, i1, int(end[i1 - 1])
        i0 = i1


def _pair_blocks(x, rows, classes, pos, max_dist, most):
    """(mask (R, C) of the block's pairs, i0, [counts (classes^2, N) per population])."""
    planes = [_planes(x[r], classes) for r in rows]
    p = torch.as_tensor(pos, device=x.device)
    k = len(classes)
    for i0, i1, j1 in _row_blocks(pos, max_dist, most):
        d = p[None, i0:j1] - p[i0:i1, None]
        mask = torch.triu(d <= max_dist, 1)
        counts = []
        for q in planes:
            c = torch.stack([(q[a, :, i0:i1].T @ q[b, :, i0:j1])[mask] for a in range(k)
                             for b in range(k)])
            counts.append(c.double())
        yield mask, d, i0, counts


def _exact_sums(x, pos, rows, bins, geno):
    """(n_bins, n_stats) sums and (n_bins,) pair counts."""
    P = len(rows)
    stats = _statistics(P, geno)
    classes, forms = ((0, 1, 2), _GENO) if geno else ((1, 0), _HAP)
    edges = torch.as_tensor(bins, device=x.device)
    nb = len(bins) - 1
    sums = torch.zeros((len(stats), nb + 2), dtype=torch.float64, device=x.device)
    cnt = torch.zeros(nb + 2, dtype=torch.float64, device=x.device)
    most = (1 << 24) // (1 if P < 3 else 2)
    for mask, d, _, counts in _pair_blocks(x, rows, classes, pos, bins[-1], most):
        b = torch.bucketize(d[mask], edges, right=True)
        one = torch.nn.functional.one_hot(b, nb + 2).double()
        pops = [_Pop(c, forms) for c in counts]
        for k in range(0, len(stats), 16):
            sums[k:k + 16] += torch.stack([_mean(pops, t) for t in stats[k:k + 16]]) @ one
        cnt += one.sum(0)
        del one, pops
    return sums[:, 1:-1].T.cpu().numpy(), cnt[1:-1].cpu().numpy()


def _het(alt, total):
    out = []
    for i in range(len(alt)):
        for j in range(i, len(alt)):
            a, b, m, n = alt[i], alt[j], total[i], total[j]
            v = 2 * (m - a) * a / (m * (m - 1)) if i == j else ((m - a) * b + a * (n - b)) / (m * n)
            out.append(float(v.sum()))
    return np.array(out)


def _hap_pair(c):
    """D numerator and the r^2 of joint haplotype counts (4, N)."""
    x = c[0] * c[3] - c[1] * c[2]
    n = c.sum(0)
    pa, pb = c[0] + c[1], c[0] + c[2]
    den = pa * (n - pa) * pb * (n - pb)
    return torch.where(den > 0, x * x / den.clamp(min=1), torch.full_like(x, math.nan))


def _window_blocks(s, most):
    """(window, sites, first row, mask (R, C) of the pairs a < b, their counts (4, N),
    carrier and valid counts of the window's sites) of every window's segregating sites."""
    x = s["hap"]
    car, val = (x == 1).sum(0), (x >= 0).sum(0)
    seg = ((car > 0) & (car < val)).nonzero().flatten()
    at = seg.cpu().numpy()
    for w, (lo, hi) in enumerate(zip(np.searchsorted(at, s["start"]),
                                     np.searchsorted(at, s["stop"]))):
        site = seg[lo:hi]
        q = _planes(x[:, site], (1, 0))
        m = int(hi - lo)
        step = max(1, most // max(1, m))
        for r in range(0, m, step):
            e = min(m, r + step)
            mask = torch.triu(torch.ones((e - r, m - r), dtype=torch.bool, device=x.device), 1)
            c = torch.stack([(q[a, :, r:e].T @ q[b, :, r:])[mask] for a in (0, 1)
                             for b in (0, 1)]).double()
            yield w, m, r, mask, c, car[site].double(), val[site].double()


def _exact_zns(s):
    """Mean DD / pi2 numerator ratio of each window's pairs with four valid haplotypes."""
    W = len(s["start"])
    tot, cnt = np.zeros(W), np.zeros(W)
    dd, _, pi = _statistics(1, False)
    for w, _, _, _, c, _, _ in _window_blocks(s, 1 << 24):
        p = [_Pop(c, _HAP)]
        num, den = _mean(p, dd), _mean(p, pi)
        ok = p[0].n >= 4
        v = torch.where(ok & (den != 0), num / torch.where(den != 0, den, 1.0), 0.0)
        tot[w] += float(v.sum())
        cnt[w] += float(ok.sum())
    return np.where(cnt > 0, tot / np.maximum(cnt, 1), 0.0)


def _exact_omega(s):
    """Largest within / across ratio of mean naive r^2 over each window's splits."""
    out = np.zeros(len(s["start"]))
    full = {}
    for w, m, r, mask, c, car, val in _window_blocks(s, 1 << 24):
        n, p = c.sum(0), car / val
        i, j = mask.nonzero(as_tuple=True)
        pi, pj = p[r + i], p[r + j]
        d = torch.where(n > 0, c[0] / n.clamp(min=1), 0.0) - pi * pj
        full.setdefault(w, torch.zeros((m, m), dtype=torch.float64, device=c.device))
        full[w][r + i, r + j] = d * d / (pi * (1 - pi) * pj * (1 - pj))
        if r + mask.shape[0] < m:
            continue
        v = full.pop(w)
        rows, cols = v.sum(1).cpu().numpy(), v.sum(0).cpu().numpy()
        for l in range(3, m - 1):
            left, cross = cols[:l].sum(), rows[:l].sum() - cols[:l].sum()
            if cross > 0:
                within = (left + rows[l:].sum()) / (l * (l - 1) // 2 + (m - l) * (m - l - 1) // 2)
                out[w] = max(out[w], within / (cross / (l * (m - l))))
    return out


def exact(case, seed):
    """run()'s outputs in 64 bits; None where a value is a whole number."""
    s = prepare(case, seed)
    kind = case["kind"]
    pos = s["pos"].cpu().numpy().astype(np.float64)
    if kind in ("two_pops", "one_pop"):
        x = s["hap"]
        keep = (((x == 0).sum(0) > 0) & ((x == 1).sum(0) > 0)).nonzero().flatten()
        x, pos = x[:, keep], pos[keep.cpu().numpy()]
        sums, cnt = _exact_sums(x, pos, list(s["sets"].values()), s["bins"], False)
        return sums if case["raw"] else np.where(cnt[:, None] > 0,
                                                 sums / np.maximum(cnt[:, None], 1), 0.0)
    if kind in ("moments_hap", "moments_geno"):
        geno = kind == "moments_geno"
        x, rows = s["geno" if geno else "hap"], list(s["sets"].values())
        alt = [x[r].clamp(min=0).sum(0).double() for r in rows]
        valid = [(x[r] >= 0).sum(0).double() for r in rows]
        total = [2 * v for v in valid] if geno else [torch.full_like(a, len(r))
                                                     for a, r in zip(alt, rows)]
        if geno:
            # sites polymorphic across the union of the populations
            a, v = sum(alt), sum(valid)
            keep = ((a > 0) & (a < 2 * v) & (v >= 2)).nonzero().flatten()
            sums, _ = _exact_sums(x[:, keep], pos[keep.cpu().numpy()], rows, s["bins"], True)
        else:
            sums, _ = _exact_sums(x, pos, rows, s["bins"], False)
        return [*sums, _het(alt, total)]
    if kind in ("hap_band", "geno_band"):
        geno = kind == "geno_band"
        x = s["geno" if geno else "hap"]
        dd, dz, pi = _statistics(1, geno)
        out = []
        for _, _, _, (c,) in _pair_blocks(x, [slice(None)], (0, 1, 2) if geno else (1, 0), pos,
                                          case["max_kb"] * 1000, 1 << 24):
            p = [_Pop(c, _GENO if geno else _HAP)]
            if geno:
                r = _rogers_huff(c)
                r2 = r * r
            else:
                r2 = _hap_pair(c)
            four = [torch.where(p[0].n >= 4, _mean(p, t), 0.0) for t in (dd, dz, pi)]
            out.append(torch.stack([r2, *four], 1))
        return None, None, torch.cat(out)
    if kind == "zns":
        return _exact_zns(s)
    if kind == "omega":
        return _exact_omega(s)
    if kind == "chunks":
        stats = _statistics(2, False)
        out, d = [], case["max_kb"] * 1000
        for i, j in _pair_chunks(pos, d, case["chunk"]):
            pops = []
            for rows in s["sets"].values():
                q = _planes(s["hap"][rows], (1, 0))
                pops.append(_Pop(torch.stack([(q[a][:, i] * q[b][:, j]).sum(0) for a in (0, 1)
                                              for b in (0, 1)]).double(), _HAP))
            out.append((None, None, None, None, torch.stack([_mean(pops, t) for t in stats], 1)))
        return out
    if kind == "rogers_huff":
        out = [_rogers_huff(c) for _, _, _, (c,) in _pair_blocks(
            s["geno"], [slice(None)], (0, 1, 2), pos, math.inf, 1 << 24)]
        return torch.cat(out)
    if kind == "r2_decay":
        r2, b = [], []
        edges = torch.as_tensor(s["bins"], device="cuda")
        for mask, d, _, (c,) in _pair_blocks(s["hap"], [slice(None)], (1, 0), pos, math.inf,
                                             1 << 24):
            r2.append(_hap_pair(c))
            b.append(torch.bucketize(d[mask], edges, right=True))
        r2, b = torch.cat(r2).cpu().numpy(), torch.cat(b).cpu().numpy()
        r2, b = r2[~np.isnan(r2)], b[~np.isnan(r2)]
        parts = [r2[b == k] for k in range(1, len(s["bins"]))]
        return np.array([np.percentile(v, [50, 90]) if len(v) else [math.nan] * 2
                         for v in parts]), None
    out = []
    for _, _, _, (c,) in _pair_blocks(s["hap"], [slice(None)], (1, 0), pos, math.inf, 1 << 24):
        p = [_Pop(c, _HAP)]
        out.append(torch.stack([_mean(p, t) for t in _statistics(1, False)] + [_hap_pair(c)]))
    dd, dz, pi, r2 = torch.cat(out, 1)
    return None, None, dict(dd=dd, dz=dz, pi2=pi, r_squared=r2)


def _rogers_huff(c):
    """Correlation of the dosages of joint genotype counts (9, N)."""
    n = c.sum(0)
    a = torch.tensor([k // 3 for k in range(9)], dtype=torch.float64, device=c.device)
    b = torch.tensor([k % 3 for k in range(9)], dtype=torch.float64, device=c.device)
    sa, sb = a @ c, b @ c
    va, vb = n * ((a * a) @ c) - sa * sa, n * ((b * b) @ c) - sb * sb
    ok = (va > 0) & (vb > 0)
    cov = n * ((a * b) @ c) - sa * sb
    return torch.where(ok, cov / torch.sqrt(torch.where(ok, va * vb, 1.0)), math.nan)


def _pair_chunks(pos, max_dist, chunk):
    """Index pairs within max_dist in anchor blocks: block k ends at the first
    anchor whose cumulative pair count reaches k * chunk."""
    m = len(pos)
    per = np.searchsorted(pos, pos + max_dist, side="right") - np.arange(m) - 1
    cum = np.cumsum(per)
    lo = 0
    for k in itertools.count(1):
        if lo >= m or (lo and cum[lo - 1] >= cum[-1]):
            return
        hi = min(m, int(np.searchsorted(cum, min(k * chunk, cum[-1]))) + 1)
        if hi <= lo:
            continue
        i = np.repeat(np.arange(lo, hi), per[lo:hi])
        start = np.repeat(np.cumsum(per[lo:hi]) - per[lo:hi], per[lo:hi])
        j = i + 1 + np.arange(len(i)) - start
        if len(i):
            yield torch.as_tensor(i, device="cuda"), torch.as_tensor(j, device="cuda")
        lo = hi
