"""All-pairs kernels and the float64 statistics kernels: exact counts, the exact
quotients of their integers (one rounding), Rogers-Huff r bit for bit."""
import numpy as np
import pytest

from oracle import ld_oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pg_gpu_gb300 import _geno, _lib as L, _ops  # noqa: E402


def np_(t):
    return t.cpu().numpy()


# SNPs: below, at and above a tile; haplotypes: one word, a chunk of words, more
@pytest.mark.parametrize("M", [1, 2, 32, 33, 97])
@pytest.mark.parametrize("H,missing,other", [(1, 0.0, 0.0), (33, 0.1, 0.0), (1024, 0.02, 0.0),
                                             (1100, 0.0, 0.05), (70, 0.1, 0.05)])
def test_tally(M, H, missing, other):
    rng = np.random.default_rng(M * H)
    x = rng.integers(0, 2, (H, M)).astype(np.int8)
    x[rng.random(x.shape) < other] = 2
    x[rng.random(x.shape) < missing] = -1
    pk = _ops.pack(torch.as_tensor(x, device="cuda"))
    c, nv = _ops.tally(pk)
    i, j = np.triu_indices(M, 1)
    want, wnv = O.counts_for_pairs(x, i, j)
    assert np.array_equal(np_(c), want.reshape(-1, 4))
    assert (nv is None) == (wnv is None)
    if nv is not None:
        assert np.array_equal(np_(nv), wnv)


@pytest.mark.parametrize("m,n", [(1, 5), (2, 3), (32, 31), (33, 33), (70, 1030), (65, 8192)])
def test_rogers_huff(m, n):
    rng = np.random.default_rng(m + n)
    g = rng.binomial(2, rng.beta(0.3, 0.3, m), (n, m)).astype(np.int8)
    g[:, 0] = 1  # no variance
    gd = torch.as_tensor(g, device="cuda")
    got = _ops.rogers_huff_all(_ops.pack_geno(gd))
    i, j = torch.triu_indices(m, m, 1, device="cuda").to(torch.int32)
    want = _geno.rh_pairs(gd, i, j) if m > 1 else got
    assert torch.equal(torch.nan_to_num(got, nan=9.0), torch.nan_to_num(want, nan=9.0))


# sample sizes: below four (zero denominators), ordinary, numerators above 53 bits;
# counts rows that 16-byte loads may and may not read
@pytest.mark.parametrize("n", [3, 60, 1000, 20_000])
@pytest.mark.parametrize("pad", [0, 1])
def test_single_terms_and_tables(n, pad):
    rng = np.random.default_rng(n + pad)
    N = 700
    c = rng.multinomial(n, [0.4, 0.2, 0.3, 0.1], (2, N)).astype(np.int32)
    c[:, ::7, 1] = 0
    c[:, ::11, :3] = 0
    buf = torch.zeros((N, 8 + pad), dtype=torch.int32, device="cuda")
    buf[:, :8] = torch.as_tensor(np.concatenate([c[0], c[1]], 1))
    views = [buf[:, :4], buf[:, 4:8]]
    nv = [None, torch.as_tensor(c[1].sum(1).astype(np.int32), device="cuda")]
    one = [L.DD_II, L.DZ_III, L.PI2_IIII, L.R, L.R2, L.DPRIME]
    two = [L.DD_IJ, L.DZ_IIJ, L.DZ_IJI, L.DZ_IJJ, L.PI2_TRIPLE, L.PI2_IIKK, L.PI2_IIKK_SYM,
           L.PI2_IJIJ]
    for kind in one + two:
        for roles in ((0, 1), (1, 0)):
            r = roles[:1] if kind in one else roles
            # a list of two terms takes the general kernel
            want = _ops.stats(views, nv, [(0, kind, r, 1.0), (1, kind, r, 0.5)], 2)[:, 0]
            got = _ops.stats(views, nv, [(0, kind, r, 1.0)], 1)[:, 0]
            assert torch.equal(torch.nan_to_num(got, nan=7.5), torch.nan_to_num(want, nan=7.5)), kind
    from pg_gpu_gb300.ld_pipeline import spec_terms
    for P, S in ((1, 3), (2, 15)):
        got = np_(_ops.stats(views[:P], nv[:P], spec_terms(P), S))
        # with a column more the list is not the table; the averages of two
        # quotients differ from one quotient by roundings of the larger
        more = spec_terms(P) + [(S, L.DD_II, (0,), 1.0)]
        want = np_(_ops.stats(views[:P], nv[:P], more, S + 1))[:, :S]
        np.testing.assert_allclose(got, want, rtol=1e-14, atol=1e-15 * np.abs(want).max())


def test_rogers_huff_on_two_streams():
    """Calls on two streams of one handle: each has its own table of sites."""
    rng = np.random.default_rng(12)
    m, n = 9000, 400
    packs = [_ops.pack_geno(torch.as_tensor(
        rng.binomial(2, rng.beta(0.3 + k, 0.5, m), (n, m)).astype(np.int8), device="cuda")) for k in range(2)]
    want = [_ops.rogers_huff_all(pk) for pk in packs]
    streams = [torch.cuda.Stream() for _ in packs]
    torch.cuda.synchronize()
    got = []
    for _ in range(3):
        for pk, s in zip(packs, streams):
            with torch.cuda.stream(s):
                got.append(_ops.rogers_huff_all(pk))
    torch.cuda.synchronize()
    for k, r in enumerate(got):
        assert torch.equal(torch.nan_to_num(r, nan=9.0), torch.nan_to_num(want[k % 2], nan=9.0))


def test_rogers_huff_entry_with_its_own_sites():
    from pg_gpu_gb300 import _lib as L
    rng = np.random.default_rng(4)
    pk = _ops.pack_geno(torch.as_tensor(rng.integers(0, 3, (50, 70)).astype(np.int8), device="cuda"))
    out = torch.empty(70 * 69 // 2, dtype=torch.float64, device="cuda")
    h = L.handle()
    L.check(L.lib().pgld_geno_rogers_huff(h, L.ptr(pk.planes), pk.n_words, pk.n_rows, 70, L.ptr(out),
                                          L.stream_ptr()), h)
    assert torch.equal(out, _ops.rogers_huff_all(pk))


# where the largest denominators of a table come near 2^63: the table's kernel and
# the general one see the same integers
@pytest.mark.parametrize("n", [38_000, 46_300, 46_400, 50_000, 55_000])
def test_table_at_the_largest_sample_sizes(n):
    from pg_gpu_gb300.ld_pipeline import spec_terms
    rng = np.random.default_rng(n)
    c = [torch.as_tensor(rng.multinomial(n, rng.dirichlet(np.full(4, 0.7), 500)).astype(np.int32),
                         device="cuda") for _ in range(2)]
    got = np_(_ops.stats(c, [None, None], spec_terms(2), 15))
    want = np_(_ops.stats(c, [None, None], spec_terms(2) + [(15, 0, (0,), 1.0)], 16))[:, :15]
    assert np.all(np.abs(got - want) <= 1e-14 * np.abs(want) + 1e-15 * np.abs(want).max(0))
    x = [v.cpu().numpy().astype(object) for v in c]
    (a1, a2, a3, a4), (b1, b2, b3, b4) = (tuple(v.T) for v in x)
    # Dz_0_0_1 against exact integers
    D, dA, dB = a1 * a4 - a2 * a3, a3 + a4 - a1 - a2, a2 + a4 - a1 - a3
    num = D * (dA * (b2 + b4 - b1 - b3) + dB * (b3 + b4 - b1 - b2))
    exact = np.array([float(v) for v in num]) / float(2 * n * n * (n - 1) * (n - 2))
    np.testing.assert_allclose(got[:, 4], exact, rtol=1e-14)
