"""Form of the genotype binned sums when the tensor cores' operands do not fit:
several populations take the popcount form, which needs none; one population,
and a form that was asked for, report the error."""
import types

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from pg_gpu_gb300 import _ops  # noqa: E402
from pg_gpu_gb300._lib import PgldError  # noqa: E402


@pytest.fixture
def calls(monkeypatch):
    """The forms that the library is asked for; the tensor-core one fails with codes[0]."""
    seen, codes = [], [-6]

    def form_of(*args):
        seen.append(args[9])
        return codes[0] if args[9] == _ops.L.FORM_TC else 0

    lib = types.SimpleNamespace(pgld_geno_binned_sums_form=form_of, pgld_last_error=lambda h: b"stub")
    monkeypatch.setattr(_ops.L, "lib", lambda: lib)
    monkeypatch.setattr(_ops.L, "handle", lambda: 0)
    monkeypatch.setattr(_ops.L, "stream_ptr", lambda: 0)
    return seen, codes


def packs(P):
    z = torch.zeros((4, 3), dtype=torch.int32)
    return [_ops.PackedGeno(z, z[:, :1], 1, 20, 4, False, False) for _ in range(P)]


def sums(P, **kw):
    return _ops.geno_binned_sums(packs(P), torch.arange(4, dtype=torch.float64), np.array([0.0, 2, 4]), **kw)


@pytest.mark.parametrize("P", [2, 3, 4])
@pytest.mark.parametrize("code", [-6, -3])
def test_several_populations_take_the_popcount_form(calls, P, code):
    seen, codes = calls
    codes[0] = code
    assert sums(P)[0].shape == (2, {2: 15, 3: 45, 4: 105}[P])
    assert seen == [1, 0]


@pytest.mark.parametrize("P,kw,code", [(1, {}, -6), (2, dict(form="tc"), -6), (2, {}, -2), (3, {}, -5)])
def test_other_errors_are_reported(calls, P, kw, code):
    seen, codes = calls
    codes[0] = code
    with pytest.raises(PgldError) as e:
        sums(P, **kw)
    assert e.value.code == code and seen == [1]
