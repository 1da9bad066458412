"""Flag pairs of several packing launches: a copy on the host must not outlive
the next launch that takes a pair."""
import pytest

torch = pytest.importorskip("torch")

from pg_gpu_gb300 import _ops  # noqa: E402


def test_flags_read_between_launches(monkeypatch):
    monkeypatch.setattr(torch.Tensor, "cpu", torch.Tensor.clone)  # a copy, as from a device
    flags = _ops.PackFlags(3, "cpu")
    flags.pair(0).copy_(torch.tensor([1, 0]))
    assert flags.read(0) == (True, False)
    flags.pair(1).copy_(torch.tensor([1, 1]))
    flags.pair(2).copy_(torch.tensor([0, 1]))
    assert [flags.read(k) for k in range(3)] == [(True, False), (True, True), (False, True)]
