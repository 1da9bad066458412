"""Order statistics of segments by radix selection: exact values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pg_gpu_gb300 import _ops  # noqa: E402

CHUNK = 1 << 15


# segments of one value, below, at and above a chunk, empty ones; many equal
# values, values that differ in the last bits only, more targets per segment
# than histograms per block
@pytest.mark.parametrize("sizes,kind", [([1, 0, 7, CHUNK], "spread"), ([CHUNK + 1, 0, 3], "spread"),
                                        ([3 * CHUNK + 5, 100], "ties"), ([5000, 2 * CHUNK - 1], "close"),
                                        ([40, 41, 42, 43, 44, 45], "r2")])
def test_segment_kth(sizes, kind):
    rng = np.random.default_rng(sum(sizes))
    n = sum(sizes)
    if kind == "spread":
        v = np.exp(rng.uniform(-300, 5, n))
    elif kind == "ties":
        v = rng.choice([0.0, 0.25, 1.0, 5e-324], n)
    elif kind == "close":
        v = (np.float64(0.3).view(np.int64) + rng.integers(0, 300, n)).view(np.float64)
    else:
        v = rng.random(n) ** 4
    off = np.concatenate([[0], np.cumsum(sizes)])
    targets, want = [], []
    for s, m in enumerate(sizes):
        if m == 0:
            continue
        order = np.sort(v[off[s]:off[s + 1]])
        for k in sorted({0, m // 2, min(m - 1, m // 2 + 1), m // 10, (9 * m) // 10, m - 1}):
            targets.append((s, k))
            want.append(order[k])
    mix = rng.permutation(len(targets))
    got = _ops.segment_kth(torch.as_tensor(v, device="cuda"), sizes, [targets[k] for k in mix])
    assert np.array_equal(got, np.asarray(want)[mix])


# segments on both sides of the length up to which a block does all passes
@pytest.mark.parametrize("sizes", [[1 << 17, 5], [(1 << 17) + 1, 1, 0, 300], [200_000, 1 << 17]])
def test_segment_kth_long(sizes):
    test_segment_kth(sizes, "ties")
    test_segment_kth(sizes, "r2")
    test_segment_kth(sizes, "close")


# whole and fractional positions: the same bins (right-open) and values
@pytest.mark.parametrize("shift", [0.0, 0.5])
def test_pairs_by_bin(shift):
    rng = np.random.default_rng(4)
    M, n = 203, 45
    x = (rng.random((n, M)) < rng.beta(0.4, 0.4, M)).astype(np.int8)
    x[rng.random(x.shape) < 0.05] = -1
    pos = np.sort(rng.choice(5000, M, replace=False)).astype(np.float64)
    pos[::2] += shift
    bins = np.array([0.0, 10, 100.5, 1000, 2000])
    pk = _ops.pack(torch.as_tensor(x, device="cuda"))
    vals, cnt = _ops.pairs_by_bin(_ops.positions_f64(pos), bins, pk=pk)
    i, j = np.triu_indices(M, 1)
    a, b = x[:, i], x[:, j]
    c = [((a == u) & (b == v)).sum(0).astype(np.int64) for u, v in ((1, 1), (1, 0), (0, 1), (0, 0))]
    m = sum(c)
    pa, pb, d = c[0] + c[1], c[0] + c[2], c[0] * c[3] - c[1] * c[2]
    den = pa * (m - pa) * pb * (m - pb)
    ok = den > 0
    r2 = np.divide(d * d, den, where=ok, out=np.zeros(len(d)))
    at = np.digitize(pos[j] - pos[i], bins) - 1
    vals, k = vals.cpu().numpy(), 0
    for b in range(len(bins) - 1):
        want = np.sort(r2[ok & (at == b)])
        assert cnt[b] == len(want)
        assert np.array_equal(np.sort(vals[k:k + cnt[b]]), want)
        k += cnt[b]
