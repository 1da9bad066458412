"""Window sums of one column equal the same column of the full call: the same
operations on the same pairs, accumulated in the same order per warp (the
float64 totals in any order: 1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pg_gpu_gb300 import _ops  # noqa: E402


@pytest.mark.parametrize("column", ["sigma_d2", "r2_naive", "dd"])
@pytest.mark.parametrize("H,missing", [(3, 0.0), (33, 0.2), (400, 0.0), (400, 0.02), (2048, 0.01)])
def test_single_columns(column, H, missing):
    rng = np.random.default_rng(H)
    M = 700
    x = (rng.random((H, M)) < rng.beta(0.4, 0.4, M)).astype(np.int8)
    x[rng.random(x.shape) < missing] = -1
    b = np.array([0, 0, 5, 5, 100, 131, 400, 640, 60], np.int64)
    e = np.array([0, 1, 5, 37, 300, 195, 640, 700, 200], np.int64)
    pk = _ops.pack(torch.as_tensor(x, device="cuda"))
    for form in ("tc", "plain"):
        whole, n = (t.cpu().numpy() for t in _ops.window_sums(pk, None, b, e, form=form))
        part, m = (t.cpu().numpy() for t in _ops.window_sums(pk, None, b, e, form=form,
                                                             columns=(column,)))
        k = _ops.WINDOW_COLUMNS.index(column)
        np.testing.assert_allclose(part[:, k], whole[:, k], rtol=1e-12,
                                   atol=1e-12 * np.abs(whole[:, k]).max())
        assert np.array_equal(m[:, [0, 2]], n[:, [0, 2]])
