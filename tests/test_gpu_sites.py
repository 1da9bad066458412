"""Per-site device passes: packing with and without a site filter, site counts,
kept-site lists and heterozygosity sums, against numpy (exact integers; the
float64 sums of at most 10^5 terms to 1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pg_gpu_gb300 import _ops  # noqa: E402


def np_(t):
    return t.cpu().numpy()


def words(bits):
    """(M, W) uint32 of an (n, M) boolean matrix, row r at bit r % 32 of word r / 32."""
    n, M = bits.shape
    W = max(1, (n + 31) // 32)
    full = np.zeros((W * 32, M), np.uint64)
    full[:n] = bits
    w = (full.reshape(W, 32, M) << np.arange(32, dtype=np.uint64)[None, :, None]).sum(1)
    return w.T.astype(np.uint32)


# rows: below, at and above a word and a block of eight words; sites: tails of
# the four-site loads and of the 128-site chunks; offset: byte alignment of the matrix
@pytest.mark.parametrize("n,M,offset", [(1, 1, 0), (31, 127, 1), (32, 128, 2), (33, 129, 3),
                                        (70, 515, 1), (255, 301, 0), (257, 64, 3), (300, 1027, 2)])
@pytest.mark.parametrize("other", [False, True])
def test_planes_and_counts(n, M, offset, other):
    rng = np.random.default_rng(n * M + offset)
    total = n + 5
    buf = torch.zeros(total * M + offset + 8, dtype=torch.int8, device="cuda")
    x = rng.integers(-1, 2, (total, M)).astype(np.int8)
    x[:, M // 2] = -1
    if M > 3:
        x[:, 1] = 1
        x[:, 3] = 0
    if other:
        x[rng.random(x.shape) < 0.05] = 3
        x[0, 0], x[-1, -1] = -7, 100
    xd = buf[offset:offset + total * M].view(total, M)
    xd.copy_(torch.as_tensor(x))
    rows = rng.permutation(total)[:n].astype(np.int32)
    y = x[rows]
    pk = _ops.pack(xd, rows)
    W = pk.n_words
    assert np.array_equal(np_(pk.planes).view(np.uint32)[:, :W], words(y == 1))
    assert np.array_equal(np_(pk.planes).view(np.uint32)[:, W:], words(y == 0))
    assert np.array_equal(np_(pk.valid).view(np.uint32), words(y >= 0))
    assert pk.has_missing == bool((y == -1).any())
    assert pk.has_other == bool(((y > 1) | (y < -1)).any())
    g = _ops.pack_geno(xd, rows)
    for v in range(3):
        assert np.array_equal(np_(g.planes).view(np.uint32)[:, v * W:(v + 1) * W], words(y == v))
    assert g.has_missing == bool((y < 0).any()) and g.has_other == bool((y > 2).any())
    if g.has_other:
        for v in range(6):
            assert np.array_equal(np_(g.ext).view(np.uint32)[:, v * W:(v + 1) * W], words(y == 3 + v))
    s, v, f = _ops.site_counts(xd, rows, flags=True)
    assert np.array_equal(np_(s), np.maximum(y, 0).astype(int).sum(0))
    assert np.array_equal(np_(v), (y >= 0).sum(0))
    assert np.array_equal(np_(f), (y == 0).any(0) * 1 + (y == 1).any(0) * 2 + (y > 1).any(0) * 4)


# sites: below, at and above the tile of the list kernel, several tiles
@pytest.mark.parametrize("M", [1, 255, 4095, 4096, 4097, 20_000])
def test_kept_sites_and_filtered_planes(M):
    rng = np.random.default_rng(M)
    x = rng.integers(-1, 3, (40, M)).astype(np.int8)
    x[:, rng.random(M) < 0.5] &= 1
    xd = torch.as_tensor(x, device="cuda")
    counts = _ops.site_counts(xd, flags=True)
    has2, a, n = (x > 1).any(0), np.maximum(x, 0).astype(int).sum(0), (x >= 0).sum(0)
    rules = {_ops.KEEP_BIALLELIC: (x == 0).any(0) & (x == 1).any(0) & ~has2,
             _ops.KEEP_SEGREGATING: (a > 0) & (a < n),
             _ops.KEEP_DIPLOID: (a > 0) & (a < 2 * n) & (n >= 2)}
    for rule, keep in rules.items():
        kept = _ops.kept_sites(rule, counts)
        assert np.array_equal(np_(kept[1]), np.nonzero(keep)[0])
        assert np.array_equal(np_(kept[0]), np.concatenate([[0], np.cumsum(keep)]))
        if not keep.any():
            continue
        got, want = _ops.pack(xd, np.arange(3, 37), kept), _ops.pack(xd[:, kept[1].long()], np.arange(3, 37))
        assert torch.equal(got.planes, want.planes) and torch.equal(got.valid, want.valid)
        assert got.has_missing == want.has_missing and got.has_other == want.has_other
        got, want = (_ops.pack_geno(xd, kept=kept), _ops.pack_geno(xd[:, kept[1].long()]))
        assert torch.equal(got.planes, want.planes)


@pytest.mark.parametrize("P,M,ploidy", [(1, 1, 1), (2, 300, 2), (3, 5000, 1), (4, 70_001, 2)])
def test_heterozygosity(P, M, ploidy):
    rng = np.random.default_rng(P + M)
    n = [20 + 7 * p for p in range(P)]
    valid = [rng.integers(2, k + 1, M) for k in n]
    alt = [rng.integers(0, ploidy * v + 1) for v in valid]
    dev = [[torch.as_tensor(t.astype(np.int32), device="cuda") for t in ts] for ts in (alt, valid)]
    got = _ops.heterozygosity(dev[0], dev[1] if ploidy == 2 else [None] * P, n, ploidy)
    m = [2.0 * v if ploidy == 2 else np.full(M, float(k)) for v, k in zip(valid, n)]
    want = []
    for i in range(P):
        for j in range(i, P):
            ri, rj = m[i] - alt[i], m[j] - alt[j]
            want.append((2 * ri * alt[i] / (m[i] * (m[i] - 1))).sum() if i == j else
                        ((ri * alt[j] + alt[i] * rj) / (m[i] * m[j])).sum())
    np.testing.assert_allclose(got, want, rtol=1e-12)


# a GenotypeMatrix does not ask for lists: rows as device tensors, arrays and lists
@pytest.mark.parametrize("form", ["device", "host", "array"])
def test_genotype_sample_sets_of_other_kinds(form):
    from pg_gpu_gb300 import moments_ld
    from pg_gpu_gb300.genotype_matrix import GenotypeMatrix
    rng = np.random.default_rng(3)
    g = torch.as_tensor(rng.binomial(2, rng.beta(0.4, 0.4, 300), (30, 300)).astype(np.int8), device="cuda")
    pos = np.sort(rng.choice(30_000, 300, replace=False))
    lists = {"pop0": list(range(14)), "pop1": list(range(10, 30))}
    to = {"device": lambda r: torch.tensor(r, device="cuda"), "host": torch.tensor, "array": np.array}[form]
    got, want = (moments_ld.compute_ld_statistics(
        genotype_matrix=GenotypeMatrix(g, pos, sample_sets=sets), use_genotypes=True,
        bp_bins=[0, 5000, 20_000], report=False)
        for sets in ({k: to(r) for k, r in lists.items()}, lists))
    for a, b in zip(got["sums"], want["sums"]):
        np.testing.assert_allclose(a, b, rtol=1e-12)


@pytest.mark.parametrize("M", [0, 1, 257, 100_001])
def test_heterozygosity_repeats_to_the_last_bit(M):
    rng = np.random.default_rng(M)
    n = [30, 41, 7]
    s = [torch.as_tensor(rng.integers(0, k + 1, M).astype(np.int32), device="cuda") for k in n]
    first = _ops.heterozygosity(s, [None] * 3, n, 1)
    assert first.shape == (6,) and (M > 0 or not first.any())
    for _ in range(30):
        assert np.array_equal(_ops.heterozygosity(s, [None] * 3, n, 1), first)


@pytest.mark.parametrize("geno", [False, True])
def test_moments_of_an_empty_population_are_refused(geno):
    from pg_gpu_gb300 import moments_ld
    from pg_gpu_gb300.genotype_matrix import GenotypeMatrix
    from pg_gpu_gb300.haplotype_matrix import HaplotypeMatrix
    x = torch.as_tensor(np.random.default_rng(2).integers(0, 2, (12, 40)).astype(np.int8), device="cuda")
    m = (GenotypeMatrix if geno else HaplotypeMatrix)(x, np.arange(40), sample_sets={"a": [0, 1, 2, 3], "b": []})
    with pytest.raises(IndexError):
        moments_ld.compute_ld_statistics(pops=["a", "b"], bp_bins=[0, 10, 20], report=False, use_genotypes=geno,
                                         **{"genotype_matrix" if geno else "haplotype_matrix": m})
