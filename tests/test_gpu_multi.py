"""Binned sums of several populations on the device: the unrolled float32
statistics (pgld_multi.cuh) against the oracle and the exact term table.

A quotient carries at most 16 float32 roundings (under 1e-6 of the absolute sum
of its terms), and the sums over lanes and steps a few more: every bin and
statistic lies within 2e-6 of the bin's sum of |x|.
"""
import numpy as np
import pytest

from oracle import ld_oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pg_gpu_gb300 import _ops  # noqa: E402

TOL = 2e-6


def np_(t):
    return t.cpu().numpy()


def panel(rng, sizes, M, top, missing):
    p = rng.beta(0.5, 0.5, M)
    x = rng.binomial(top, p, (sum(sizes), M)).astype(np.int8)
    # neighbours alike, so that the statistics do not all vanish
    for s in range(1, M):
        same = rng.random(sum(sizes)) < 0.6
        x[same, s] = x[same, s - 1]
    x[rng.random(x.shape) < missing] = -1
    edges = np.concatenate([[0], np.cumsum(sizes)])
    return x, [np.arange(a, b, dtype=np.int32) for a, b in zip(edges[:-1], edges[1:])]


# sizes: words of the concatenated populations that end inside, at and across the
# 32-word staging chunk, one haplotype, the largest float32-exact population
@pytest.mark.parametrize("sizes,M,spacing", [([30, 33, 5], 97, "int"), ([640, 650, 300], 65, "int"),
                                             ([1, 4, 1030, 32], 70, "int"),
                                             ([40, 41, 42, 43], 161, "fraction"),
                                             ([2048, 64, 100], 64, "int"),
                                             ([50, 20, 31], 130, "map")])
def test_haplotype_sums_of_three_and_four_populations(sizes, M, spacing):
    rng = np.random.default_rng(sum(sizes) + M)
    x, rows = panel(rng, sizes, M, 1, 0.03)
    pos = np.sort(rng.choice(40 * M, M, replace=False)).astype(np.float64)
    if spacing == "fraction":
        pos += 0.25
        pos[::3] += 0.5
    bc = np.cumsum(rng.uniform(0.1, 2.0, M)) if spacing == "map" else None
    bins = np.array([0.0, 3, 10, 30]) if spacing == "map" else np.array([1.0, 60, 90.5, 400, 1500])
    md = 900.0 if spacing == "map" else None
    pops = [_ops.pack(torch.as_tensor(x, device="cuda"), r) for r in rows]
    sums, cnt = _ops.binned_sums(pops, _ops.positions_f64(pos), bins, max_dist=md,
                                 bin_coord=None if bc is None else torch.as_tensor(bc, device="cuda"))
    ref, rcnt, rabs = O.binned_sums(x, pos, rows, bins, coords=bc, max_dist=md, abs_sums=True)
    assert np.array_equal(np_(cnt), rcnt) and rcnt.sum() > 500
    assert np.all(np.abs(np_(sums) - ref) <= TOL * rabs + 1e-300)
    again, _ = _ops.binned_sums(pops, _ops.positions_f64(pos), bins, max_dist=md,
                                bin_coord=None if bc is None else torch.as_tensor(bc, device="cuda"))
    np.testing.assert_allclose(np_(again), np_(sums), rtol=1e-13, atol=1e-300)


# the range call: the first SNP of a pair inside the anchors only
def test_haplotype_sums_over_an_anchor_range():
    rng = np.random.default_rng(3)
    x, rows = panel(rng, [37, 20, 64], 200, 1, 0.02)
    pos = np.sort(rng.choice(8000, 200, replace=False)).astype(np.float64)
    bins = np.array([0.0, 100, 1000, 3000])
    pops = [_ops.pack(torch.as_tensor(x, device="cuda"), r) for r in rows]
    pos_d = _ops.positions_f64(pos)
    whole, n = _ops.binned_sums(pops, pos_d, bins)
    parts = [_ops.binned_sums(pops, pos_d, bins, anchors=r) for r in ((0, 45), (45, 46), (46, 200))]
    assert np.array_equal(sum(np_(c) for _, c in parts), np_(n))
    _, _, rabs = O.binned_sums(x, pos, rows, bins, abs_sums=True)
    assert np.all(np.abs(sum(np_(s) for s, _ in parts) - np_(whole)) <= TOL * rabs)


@pytest.mark.parametrize("sizes,M,missing,spacing", [([30, 33], 97, 0.03, "int"),
                                                     ([5, 6], 64, 0.2, "int"),
                                                     ([3, 4, 5], 70, 0.3, "int"),
                                                     ([128, 129, 31], 65, 0.02, "fraction"),
                                                     ([9, 8, 40, 21], 100, 0.05, "map"),
                                                     ([2048, 7], 33, 0.01, "int"),
                                                     ([2060, 30], 33, 0.01, "int")])
def test_genotype_sums_match_the_term_table(sizes, M, missing, spacing):
    """Tensor-core form against the popcount form, which evaluates the exact
    term table: small samples give the same infinities and NaN."""
    rng = np.random.default_rng(sum(sizes) + M)
    x, rows = panel(rng, sizes, M, 2, missing)
    pos = np.sort(rng.choice(40 * M, M, replace=False)).astype(np.float64)
    if spacing == "fraction":
        pos[::2] += 0.5
    bc = np.cumsum(rng.uniform(0.1, 2.0, M)) if spacing == "map" else None
    bins = np.array([0.0, 3, 10, 30]) if spacing == "map" else np.array([1.0, 60, 90.5, 400, 1500])
    md = 900.0 if spacing == "map" else None
    pops = [_ops.pack_geno(torch.as_tensor(x, device="cuda"), r) for r in rows]
    kw = dict(max_dist=md, bin_coord=None if bc is None else torch.as_tensor(bc, device="cuda"))
    pos_d = _ops.positions_f64(pos)
    got, c_got = (np_(t) for t in _ops.geno_binned_sums(pops, pos_d, bins, form="tc", **kw))
    want, c_want = (np_(t) for t in _ops.geno_binned_sums(pops, pos_d, bins, form="plain", **kw))
    assert np.array_equal(c_got, c_want) and c_want.sum() > 200
    fine = np.isfinite(want)
    assert np.array_equal(fine, np.isfinite(got))
    assert np.array_equal(np.isnan(want), np.isnan(got))
    with np.errstate(all="ignore"):
        _, _, rabs = O.geno_binned_sums(x, pos, rows, bins, coords=bc, max_dist=md, abs_sums=True)
    assert np.all(np.abs(got - want)[fine] <= (TOL * rabs + 1e-300)[fine])
