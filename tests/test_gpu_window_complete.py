"""Window sums of lists whose SNPs all have the same valid haplotypes: the same
pair values, added in the same blocks, as the general kernel forms.  The general
kernel is made to take the same windows by one more listed SNP, in no window,
with another missing haplotype (the float64 totals come in any order: 1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pg_gpu_gb300 import _ops  # noqa: E402

BEGIN = np.array([0, 0, 3, 5, 100, 131, 400, 640, 60, 7, 1, 250, 300, 9], np.int64)
END = np.array([0, 1, 5, 37, 228, 260, 655, 897, 316, 400, 900, 250, 899, 10], np.int64)


@pytest.mark.parametrize("columns", [("sigma_d2",), ("r2_naive",), _ops.WINDOW_COLUMNS])
@pytest.mark.parametrize("H,absent", [(2, 0), (5, 1), (32, 0), (33, 0), (130, 7), (400, 0), (1025, 3),
                                      (2048, 0)])
def test_complete_lists_match_general_kernel(columns, H, absent):
    rng = np.random.default_rng(H)
    M = 900
    x = (rng.random((H, M + 1)) < rng.beta(0.3, 0.6, M + 1)).astype(np.int8)
    x[:, ::50] = 0  # monomorphic SNPs
    x[rng.choice(H, absent, replace=False), :M] = -1
    x[:, M] = -1 if absent == 0 else 1
    pk = _ops.pack(torch.as_tensor(x, device="cuda"))
    idx = rng.permutation(M).astype(np.int32)
    here, n = (t.cpu().numpy() for t in _ops.window_sums(pk, idx, BEGIN, END, form="tc", columns=columns))
    listed = np.append(idx, np.int32(M))
    ref, m = (t.cpu().numpy() for t in _ops.window_sums(pk, listed, BEGIN, END, form="tc",
                                                        columns=columns))
    for c in columns:
        k = _ops.WINDOW_COLUMNS.index(c)
        np.testing.assert_allclose(here[:, k], ref[:, k], rtol=1e-12, atol=1e-12 * np.abs(ref[:, k]).max())
    checked = [0, 1, 2] if "r2" in columns else [0, 2]
    assert np.array_equal(n[:, checked], m[:, checked])


# lists shorter than the operand's boxes, down to one SNP
@pytest.mark.parametrize("M", [1, 2, 5, 127, 130])
def test_short_lists(M):
    rng = np.random.default_rng(M)
    x = (rng.random((50, M + 1)) < 0.4).astype(np.int8)
    x[:, M] = -1
    pk = _ops.pack(torch.as_tensor(x, device="cuda"))
    b, e = np.array([0, 0], np.int64), np.array([M, M // 2], np.int64)
    got = []
    for n in (M, M + 1):
        s, c = _ops.window_sums(pk, np.arange(n, dtype=np.int32), b, e, form="tc", columns=("sigma_d2",))
        got.append((s.cpu().numpy()[:, 1], c.cpu().numpy()[:, [0, 2]]))
    np.testing.assert_allclose(got[0][0], got[1][0], rtol=1e-12, atol=1e-12 * np.abs(got[1][0]).max())
    assert np.array_equal(got[0][1], got[1][1])
