"""CP-APR's rounds driven by the host over the row-ordered stream, which is
what runs when the queued rounds cannot have their pinned poll words: the
same solve as with queued rounds.  (The bulk-copy switch selects them; ranks
without whole 16-byte rows then run the register-staged kernel.)"""
import numpy as np
import pytest

import alto_b200 as ab
from alto_b200 import synth
from test_apr_limits_gpu import _solve
from conftest import rel_fro

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("eps", [0.3, 1e-30])
@pytest.mark.parametrize("rank", [1, 3, 25])
def test_host_rounds_match_queued_rounds(monkeypatch, rank, eps):
    d, cidx, vals = synth.uniform_distinct((90, 80, 70), 30_000, seed=rank)
    at = ab.create_alto(ab.SparseTensor.from_arrays(d, cidx, np.ceil(vals * 5)), 8, 0, val_dtype="u32")
    monkeypatch.setenv("ALTOB_PHI_TMA", "1")
    got, U = _solve(monkeypatch, "rows", at, d, rank, "f64", 1, 5, eps)
    monkeypatch.setenv("ALTOB_PHI_TMA", "0")
    want, V = _solve(monkeypatch, "rows", at, d, rank, "f64", 1, 5, eps)
    assert (got["outer"], got["inner"]) == (want["outer"], want["inner"])
    assert abs(got["kkt"] - want["kkt"]) <= 1e-9 * max(1.0, abs(want["kkt"]))
    for a, b in zip(U, V):
        assert rel_fro(a, b) < 1e-9  # the order of atomic additions
