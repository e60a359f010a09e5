"""CP-APR with a limit on the inner rounds that is far above the rounds it
takes: the same solve as with a near limit, and no more device memory (the
queued rounds keep a fixed record per mode, whatever the limit)."""
import numpy as np
import pytest

import alto_b200 as ab
from alto_b200 import synth
from conftest import rel_fro

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _solve(monkeypatch, kind, at, dims, rank, prec, outer, inner, eps):
    monkeypatch.setenv("ALTOB_APR_PHI", kind)
    dt = torch.float64 if prec == "f64" else torch.float32
    U = [torch.from_numpy(u).to(dt).cuda() for u in synth.random_factors(dims, rank, seed=rank)]
    M = ab.KruskalModel([int(d) for d in dims], rank, U, torch.ones(rank, dtype=dt, device="cuda"))
    s = ab.cp_apr_alto(at, M, outer, inner, eps)
    return s, [u.double().cpu().numpy() for u in U]


@pytest.mark.parametrize("limit", [50_000_000, 2**31 - 1])
def test_far_limit_on_inner_rounds(monkeypatch, limit):
    d, cidx, vals = synth.uniform_distinct((60, 50, 40), 20_000, seed=1)
    at = ab.create_alto(ab.SparseTensor.from_arrays(d, cidx, np.ceil(vals * 5)), 8, 0, val_dtype="u32")
    four, _ = _solve(monkeypatch, "otf", at, d, 8, "f64", 1, 4, 1e-30)
    eps = four["kkt"] * (1 + 1e-6)  # what four rounds leave: met by the fourth round of every mode
    want, V = _solve(monkeypatch, "rows", at, d, 8, "f64", 1, 20, eps)
    free = torch.cuda.mem_get_info()[0]
    got, U = _solve(monkeypatch, "rows", at, d, 8, "f64", 1, limit, eps)
    assert free - torch.cuda.mem_get_info()[0] < 64 << 20
    assert (got["outer"], got["inner"]) == (want["outer"], want["inner"])
    assert abs(got["kkt"] - want["kkt"]) <= 1e-9 * max(1.0, abs(want["kkt"]))
    for a, b in zip(U, V):
        assert rel_fro(a, b) < 1e-9  # the order of atomic additions
