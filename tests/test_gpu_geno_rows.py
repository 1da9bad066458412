"""Genotype band pairs: the counts leave as whole rows in 16-byte stores with the
ends word by word, wherever the output starts; every place of the output's start
to a 16-byte boundary, bands narrower and wider than a warp, and every number of
epilogue groups (by the individuals) gives the plain form's integers, and nothing
outside the output is written."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pg_gpu_gb300 import _lib as L  # noqa: E402
from pg_gpu_gb300 import _ops  # noqa: E402


@pytest.mark.parametrize("n_ind,max_dist", [(40, 3.0), (500, 40.0), (800, 200.0), (1000, 33.0), (1100, 70.0)])
def test_counts_at_every_alignment(n_ind, max_dist):
    rng = np.random.default_rng(n_ind)
    M = 131
    g = rng.integers(0, 3, (n_ind, M)).astype(np.int8)
    g[rng.random(g.shape) < 0.05] = -1
    pk = _ops.pack_geno(torch.as_tensor(g, device="cuda"))
    pos = _ops.positions_f64(np.cumsum(rng.integers(1, 3, M)))
    want, nv, _ = _ops.geno_band_pairs(pk, pos, max_dist, form="plain", with_stats=False)
    off, n = _ops.band_offsets(pos, max_dist)
    h = L.handle()
    for shift in range(4):
        buf = torch.full((9 * n + 8,), -7, dtype=torch.int32, device="cuda")
        out = buf[shift:shift + 9 * n]
        got = torch.empty(n, dtype=torch.int32, device="cuda")
        L.check(L.lib().pgld_geno_band_pairs_at(h, ctypes.byref(_ops.geno_panel([pk])), L.ptr(pos), max_dist,
                                                L.ptr(off), L.ptr(out), L.ptr(got), None, 0, n, L.FORM_TC,
                                                L.stream_ptr()), h)
        assert torch.equal(out.view(n, 9), want) and torch.equal(got, nv)
        assert (buf[:shift] == -7).all() and (buf[shift + 9 * n:] == -7).all()
