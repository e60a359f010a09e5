"""FP32 CP-APR whose queued rounds stop midway: a tolerance well between the
violations that two neighbouring numbers of rounds leave, so that rounding
decides no count, gives the rounds and the model of the host-driven run."""
import numpy as np
import pytest

import alto_b200 as ab
from alto_b200 import synth
from conftest import rel_fro
from test_apr_limits_gpu import _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank", [8, 25])
def test_fp32_rounds_stop_midway(monkeypatch, rank):
    d, cidx, vals = synth.uniform_distinct((60, 50, 40), 20_000, seed=rank)
    at = ab.create_alto(ab.SparseTensor.from_arrays(d, cidx, np.ceil(vals * 5)), 8, 0, val_dtype="u32")
    left = [_solve(monkeypatch, "otf", at, d, rank, "f64", 1, k, 1e-30)[0]["kkt"] for k in range(2, 9)]
    k = max(range(len(left) - 1), key=lambda i: left[i] / left[i + 1])
    assert left[k] > 1.02 * left[k + 1]  # FP32 rounding moves a violation by about 1e-5 of its value
    eps = (left[k] * left[k + 1]) ** 0.5
    got, U = _solve(monkeypatch, "rows", at, d, rank, "f32", 1, 20, eps)
    want, V = _solve(monkeypatch, "otf", at, d, rank, "f32", 1, 20, eps)
    assert 3 < got["inner"] < 3 * 20
    assert (got["outer"], got["inner"]) == (want["outer"], want["inner"])
    for a, b in zip(U, V):
        assert rel_fro(a, b) < 2e-3  # the tolerance of the FP32 rounds' other tests
