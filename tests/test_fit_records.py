"""The harness's packed parameter records: what the loss hands to the adjoint is with_theta of each record and its
row, whatever the shapes.  No GPU."""
import ctypes as C

import numpy as np
import pytest

from artful_gb300 import capi, fit


class Recorder:
    """In the adjoint's place: keeps what it was called with."""

    def __call__(self, params, targets):
        self.params = [bytes(p) for p in fit.packed(params)]
        return np.zeros(len(params)), np.zeros((len(params), 5)), None


def _records(n):
    return [fit.hole_params(0.1 + 0.1 * k, 0.9, 1.0 + 0.1 * k, 3.0, 30.0 + k, seed=k) for k in range(n)]


@pytest.mark.parametrize("rows", [1, 3, 4, 7])
@pytest.mark.parametrize("columns", [1, 4, 5, 6])
@pytest.mark.parametrize("kind", ["list", "tuple", "array", "generator"])
def test_rows_and_records_go_together(lib, rows, columns, kind):
    import torch
    records = _records(4)
    base = {"list": records, "tuple": tuple(records), "array": (capi.HoleParams * 4)(*records),
            "generator": (r for r in records)}[kind]
    theta = torch.linspace(0.1, 0.9, rows * columns).reshape(rows, columns)
    adjoint = Recorder()
    loss = fit.hole_loss().apply(theta, adjoint, base, None)
    want = [bytes(fit.with_theta(r, t)) for r, t in zip(records, theta.numpy())]
    assert adjoint.params == want and len(loss) == len(want)
    assert [bytes(r) for r in records] == [bytes(r) for r in _records(4)]  # (the caller's records stay as they are)


@pytest.mark.parametrize("shape", [(), (5,), (1, 4, 5)])
def test_a_theta_without_rows_is_refused(lib, shape):
    import torch
    with pytest.raises(TypeError):
        fit.hole_loss().apply(torch.zeros(shape), Recorder(), _records(4), None)


def test_other_arrays_are_not_taken_for_records(lib):
    with pytest.raises(TypeError):
        fit.packed((C.c_double * 3)(1.0, 2.0, 3.0))
    assert len(fit.packed([])) == 0
