"""Row lists of several populations: checked before they become 32-bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from pg_gpu_gb300 import _ops  # noqa: E402


@pytest.fixture(autouse=True)
def on_host(monkeypatch):
    monkeypatch.setattr(_ops.L, "as_device", lambda x, dtype=None: torch.as_tensor(np.asarray(x)))


@pytest.mark.parametrize("bad", [[2 ** 32 + 1], [2 ** 32], [-2 ** 32], [1 - 2 ** 32], [10], [-1]])
@pytest.mark.parametrize("at", [0, 1])
def test_rows_out_of_range_are_refused(bad, at):
    lists = [[0, 1], [3, 9]]
    lists[at] = lists[at] + bad
    with pytest.raises(IndexError):
        _ops.device_rows(lists, 10)


def test_rows_of_every_list():
    lists = [[4, 0, 9], [], np.array([7, 7], np.uint8), torch.tensor([1, 2])]
    got = _ops.device_rows(lists, 10)
    assert [r.tensor.tolist() for r in got] == [[4, 0, 9], [], [7, 7], [1, 2]]
    assert all(r.tensor.dtype == torch.int32 for r in got)
