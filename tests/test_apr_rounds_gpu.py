"""CP-APR's inner rounds queued without the host (row-ordered Phi) against
the host-driven rounds of the on-the-fly Phi: the same number of rounds when
the violation meets the tolerance midway, the same model, for streams shorter
than a warp's range, of one range, and of many, every lane layout and both
types; and bench mode (all rounds)."""
import numpy as np
import pytest

import alto_b200 as ab
from alto_b200 import synth
from conftest import rel_fro

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _solve(monkeypatch, kind, at, dims, rank, prec, outer, inner, eps, bench):
    monkeypatch.setenv("ALTOB_APR_PHI", kind)
    dt = torch.float64 if prec == "f64" else torch.float32
    U = [torch.from_numpy(u).to(dt).cuda() for u in synth.random_factors(dims, rank, seed=rank)]
    M = ab.KruskalModel([int(d) for d in dims], rank, U, torch.ones(rank, dtype=dt, device="cuda"))
    s = ab.cp_apr_alto(at, M, outer, inner, eps, dobench=bench)
    return s, [u.double().cpu().numpy() for u in U]


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("rank", [1, 3, 8, 16, 33, 64, 100])
@pytest.mark.parametrize("nnz", [1, 31, 33, 3_000, 200_000])
def test_queued_rounds_match_host_rounds(monkeypatch, nnz, rank, prec):
    dims = (90, 80, 70)
    d, cidx, vals = synth.uniform_distinct(dims, nnz, seed=nnz)
    at = ab.create_alto(ab.SparseTensor.from_arrays(d, cidx, np.ceil(vals * 5)), 8, 0, val_dtype="u32")
    # FP64: a tolerance that some modes meet before their last round; FP32: none
    # does, so rounding decides no count.  One outer iteration outside bench
    # mode: a second one is compared with the first for exact equality of the
    # violation, which at rank 1 is rounding alone.
    eps = 0.3 if prec == "f64" else 1e-30
    for bench in (False, True):
        got, U = _solve(monkeypatch, "rows", at, d, rank, prec, 2 if bench else 1, 5, eps, bench)
        want, V = _solve(monkeypatch, "otf", at, d, rank, prec, 2 if bench else 1, 5, eps, bench)
        assert (got["outer"], got["inner"]) == (want["outer"], want["inner"])
        # sums of a Phi row in another order, through at most 10 rounds of 3 modes
        tol = 1e-9 if prec == "f64" else 2e-3
        assert abs(got["kkt"] - want["kkt"]) <= tol * max(1.0, abs(want["kkt"]))
        for a, b in zip(U, V):
            assert rel_fro(a, b) < tol, (bench, rel_fro(a, b))
    if nnz == 200_000 and prec == "f64":
        assert got["inner"] == 30  # bench mode ran every round


def test_rounds_stop_midway(monkeypatch):
    """The tolerance is the violation that four host-driven rounds leave, so
    every mode of the first outer iteration stops by its fourth round of 20."""
    d, cidx, vals = synth.uniform_distinct((60, 50, 40), 20_000, seed=1)
    at = ab.create_alto(ab.SparseTensor.from_arrays(d, cidx, np.ceil(vals * 5)), 8, 0, val_dtype="u32")
    four, _ = _solve(monkeypatch, "otf", at, d, 8, "f64", 1, 4, 1e-30, False)
    eps = four["kkt"] * (1 + 1e-6)
    got, _ = _solve(monkeypatch, "rows", at, d, 8, "f64", 1, 20, eps, False)
    want, _ = _solve(monkeypatch, "otf", at, d, 8, "f64", 1, 20, eps, False)
    assert 0 < got["inner"] <= 3 * 4
    assert (got["outer"], got["inner"]) == (want["outer"], want["inner"])
    assert abs(got["loglik"] - want["loglik"]) <= 1e-9 * abs(want["loglik"])
    # met at once: one round per mode
    one, _ = _solve(monkeypatch, "rows", at, d, 8, "f64", 2, 20, 1e300, False)
    assert one["inner"] == 3 * one["outer"]
