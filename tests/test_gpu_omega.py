"""omega of batched windows from their row and column sums on the device, against
the host's prefix sums (float64 sums in another order, of terms up to 10^5 times
the sum across a split: 1e-9)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pg_gpu_gb300 import _ops  # noqa: E402


# window sizes: below the smallest with a split, at and around the 256-split
# block, several blocks; negative sums as sigma_D^2 has them
@pytest.mark.parametrize("sizes", [[0, 1, 4, 5, 6], [255, 256, 257, 258, 259], [3000, 0, 511, 12]])
@pytest.mark.parametrize("shift", [0.0, -0.4, -2.0])
def test_window_omega(sizes, shift):
    rng = np.random.default_rng(sum(sizes))
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    rows, cols, want = [], [], []
    for m in sizes:
        r2 = np.triu(rng.random((m, m)) + shift, 1)
        rows.append(r2.sum(1))
        cols.append(r2.sum(0))
        want.append(_ops.omega_from_sums(rows[-1], cols[-1]))
    begin = off[:-1] + 7
    got = _ops.window_omega(torch.as_tensor(np.concatenate(rows), device="cuda"),
                            torch.as_tensor(np.concatenate(cols), device="cuda"), off, begin,
                            begin + np.asarray(sizes))
    np.testing.assert_allclose(got, want, rtol=1e-9)
