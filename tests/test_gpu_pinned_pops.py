"""Several populations of a matrix in pinned host memory: flags, planes and sums
equal those of the device matrix, population by population."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pg_gpu_gb300 import _ops  # noqa: E402
from pg_gpu_gb300.haplotype_matrix import HaplotypeMatrix  # noqa: E402

BINS = np.logspace(3, 5, 7)


def panel(clean, pops, M=700, n=40):
    """Populations of n haplotypes, those not in `clean` with codes -1 and 2."""
    rng = np.random.default_rng(10 * pops + clean)
    hap = (rng.random((pops * n, M)) < rng.beta(0.4, 0.4, M)).astype(np.int8)
    for p in range(pops):
        if p != clean:
            part = hap[p * n:(p + 1) * n]
            part[rng.random(part.shape) < 0.03] = -1
            part[rng.random(part.shape) < 0.02] = 2
    pos = np.sort(rng.choice(300_000, M, replace=False)).astype(np.int64)
    return hap, pos, {f"p{k}": list(range(k * n, (k + 1) * n)) for k in range(pops)}


@pytest.mark.parametrize("clean", [0, 1])
def test_two_populations_with_other_codes(clean):
    hap, pos, sets = panel(clean, 2)
    hm = HaplotypeMatrix(torch.as_tensor(hap).pin_memory(), pos, sample_sets=sets)
    ref = HaplotypeMatrix(torch.as_tensor(hap, device="cuda"), pos, sample_sets=sets)
    for ac in (False, True):
        got, want = (m.compute_ld_statistics_gpu_two_pops(BINS, "p0", "p1", raw=True, ac_filter=ac)
                     for m in (hm, ref))
        for key in want:
            a, b = (np.array(list(d[key].values())) for d in (got, want))
            # the same float32 partial sums, added in any order: at most 2,000 to a
            # bin's slot, of 2.4e5 pairs of magnitude at most 1
            np.testing.assert_allclose(a, b, rtol=0, atol=2000 * 2.0 ** -53 * 2.4e5)
    assert hm.device == "CPU"
    for k in range(2):
        pk = hm.packed(f"p{k}")
        assert (pk.has_missing, pk.has_other) == (k != clean,) * 2
        (c, nv), (rc, rnv) = (m.tally_gpu_haplotypes(f"p{k}") for m in (hm, ref))
        assert torch.equal(c, rc) and (nv is None) == (rnv is None) == (k == clean)
        assert nv is None or torch.equal(nv, rnv)


@pytest.mark.parametrize("pops", [3, 4])
def test_flags_of_several_populations(pops):
    hap, pos, sets = panel(0, pops)
    hm = HaplotypeMatrix(torch.as_tensor(hap).pin_memory(), pos, sample_sets=sets)
    assert [(pk.has_missing, pk.has_other) for pk in hm.packed_all(list(sets))] == [
        (k != 0,) * 2 for k in range(pops)]


def test_host_matrix_is_free_after_packing():
    hap, _, sets = panel(0, 3, M=4001)
    host = torch.as_tensor(hap).pin_memory()
    want = _ops.pack_all(torch.as_tensor(hap, device="cuda"), list(sets.values()))
    got = _ops.pack_all(host, list(sets.values()))
    host.zero_()
    for a, b in zip(got, want):
        assert torch.equal(a.planes, b.planes) and torch.equal(a.valid, b.valid)
        assert (a.has_missing, a.has_other) == (b.has_missing, b.has_other)
