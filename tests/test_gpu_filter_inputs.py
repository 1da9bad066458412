"""The biallelic filter inside the binned calls on every kind of matrix that a
HaplotypeMatrix can hold: the same result as filtering first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pg_gpu_gb300 import _ops  # noqa: E402
from pg_gpu_gb300.haplotype_matrix import HaplotypeMatrix  # noqa: E402

H, M = 45, 601
BINS = np.logspace(3, 5, 7)


def panel():
    rng = np.random.default_rng(5)
    hap = (rng.random((H, M)) < rng.beta(0.3, 0.3, M)).astype(np.int8)
    hap[rng.random(hap.shape) < 0.02] = -1
    hap[:, ::7] += (rng.random((H, (M + 6) // 7)) < 0.1) * 1  # some sites with a 2
    hap[:, 3::50] = 0
    return hap, np.sort(rng.choice(250_000, M, replace=False)).astype(np.int64)


def want(hap, pos):
    """The reference value: an int8 C-ordered device matrix, filtered first."""
    hm = HaplotypeMatrix(torch.as_tensor(np.ascontiguousarray(hap), device="cuda"),
                         np.ascontiguousarray(pos))
    return hm.apply_biallelic_filter().compute_ld_statistics_gpu_single_pop(BINS, raw=True, ac_filter=False)


def same(hm, hap, pos):
    assert hm.compute_ld_statistics_gpu_single_pop(BINS, raw=True) == want(hap, pos)


def held(t, pos):
    """A device matrix that holds t as it is (the constructor would copy)."""
    hm = HaplotypeMatrix(torch.zeros((2, 2), dtype=torch.int8, device="cuda"), pos)
    hm.haplotypes = t
    return hm


@pytest.mark.parametrize("form", ["int8", "columns", "transposed", "rows", "int32", "int64", "wide"])
def test_device_matrix_as_held(form):
    hap, pos = panel()
    d = torch.as_tensor(hap, device="cuda")
    if form == "columns":
        t = d.repeat_interleave(2, 1)[:, ::2]
    elif form == "transposed":
        t = d.t().contiguous().t()
    elif form == "rows":
        t = d.repeat_interleave(3, 0)[::3]
    elif form == "wide":
        # 256 and 257 are above 1, not the 0 and 1 that their low bytes spell
        t = d.to(torch.int32)
        t[0, ::11] = 256
        t[1, ::13] = 257
        keep = ((t >= 2).sum(0) == 0).cpu().numpy()
        return same(held(t, pos), hap[:, keep], pos[keep])
    else:
        t = d.to(getattr(torch, form))
    same(held(t, pos), hap, pos)


@pytest.mark.parametrize("form", ["int8", "backwards", "fortran", "int16", "pinned", "overlap"])
def test_host_matrix(form):
    hap, pos = panel()
    if form == "backwards":
        x = hap[:, ::-1].copy()[:, ::-1]
        p = pos[::-1].copy()[::-1]
        return same(HaplotypeMatrix(x, p), hap, pos)
    if form == "pinned":
        return same(HaplotypeMatrix(torch.as_tensor(hap).pin_memory(), pos), hap, pos)
    if form == "overlap":
        # windows of one pinned row: row r starts at site r
        row = torch.as_tensor(hap.reshape(-1)[:M + H]).pin_memory()
        x = row.as_strided((H, M), (1, 1))
        return same(HaplotypeMatrix(x, pos), x.numpy(), pos)
    x = np.asfortranarray(hap) if form == "fortran" else hap.astype(form)
    same(HaplotypeMatrix(x, pos), hap, pos)


def test_site_counts_of_strided_and_wider_tensors():
    hap, _ = panel()
    d = torch.as_tensor(hap, device="cuda")
    ref = [t.cpu() for t in _ops.site_counts(d, flags=True)]
    for t in (d.repeat_interleave(2, 1)[:, ::2], d.t().contiguous().t(), d.to(torch.int32)):
        for a, b in zip(_ops.site_counts(t, flags=True), ref):
            assert torch.equal(a.cpu(), b)


# checked on the host: a gather past the end would fault on the device
@pytest.mark.parametrize("device", ["cpu", "cuda"])
def test_positions_that_end_early(device):
    hap, pos = panel()
    hap[:, -2] = 0
    hap[:, -1] = 0
    x = hap if device == "cpu" else torch.as_tensor(hap, device=device)
    same(HaplotypeMatrix(x, pos[:-1]), hap[:, :-1], pos[:-1])  # the sites without one are dropped
    hm = HaplotypeMatrix(x, pos[:M // 2])
    with pytest.raises(IndexError):
        hm.compute_ld_statistics_gpu_single_pop(BINS, raw=True)
    if device == "cuda":
        with pytest.raises(IndexError):
            hm.get_subset([M - 1])


def test_host_array_set_on_a_device_matrix():
    hap, pos = panel()
    sets = {"a": list(range(20)), "b": list(range(20, H))}
    ref = HaplotypeMatrix(torch.as_tensor(hap, device="cuda"), pos, sample_sets=sets)
    hm = HaplotypeMatrix(torch.zeros_like(ref.haplotypes), pos, sample_sets=sets)
    hm.haplotypes = hap
    got, want = ([(p.planes, p.valid) for p in m.packed_all(["a", "b"])] for m in (hm, ref))
    for a, b in zip(got, want):
        assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("ac", [True, False])
def test_pinned_matrix_changed_on_the_device(ac):
    hap, pos = panel()
    hm = HaplotypeMatrix(torch.as_tensor(hap).pin_memory(), pos)
    hm.transfer_to_gpu()
    hm.haplotypes[:, 5::9] = 0
    changed = hm.haplotypes.cpu().numpy()
    hm.transfer_to_cpu()
    got = hm.compute_ld_statistics_gpu_single_pop(BINS, raw=True, ac_filter=ac)
    ref = HaplotypeMatrix(torch.as_tensor(changed, device="cuda"), pos)
    assert got == ref.compute_ld_statistics_gpu_single_pop(BINS, raw=True, ac_filter=ac)
