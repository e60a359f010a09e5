"""tt_logLikelihood at the edges of its lane layouts: ranks below, at and past
one lane group's row, vector and scalar rows, misaligned factors, orders 2 to
5, nonzero counts around a warp's 32, every stored value type."""
import numpy as np
import pytest

import alto_b200 as ab
from alto_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _reference(cidx, vals, U, lam, eps):
    U = [u.astype(np.float64) for u in U]
    p = np.ones((cidx.shape[1], U[0].shape[1]))
    for c, u in zip(cidx, U):
        p *= u[c.astype(np.int64)]
    return float((vals * np.log(np.maximum(p.sum(1), eps))).sum() - U[0].sum())


@pytest.mark.parametrize("dims", [(9, 7), (40, 30, 20), (13, 11, 9, 5), (9, 8, 7, 6, 5)])
@pytest.mark.parametrize("rank", [1, 3, 4, 8, 16, 17, 33, 36, 100])
@pytest.mark.parametrize("prec,vdt", [("f64", "f64"), ("f64", "u32"), ("f32", "f32"), ("f32", "u32")])
def test_loglik_matches_numpy(dims, rank, prec, vdt):
    for nnz in (1, 31, 33, min(1000, int(np.prod(dims)) // 2)):
        d, cidx, vals = synth.uniform_distinct(dims, nnz, seed=nnz + rank)
        vals = np.ceil(vals * 9)  # counts: exact in every stored type
        at = ab.create_alto(ab.SparseTensor.from_arrays(d, cidx, vals), 4, 0, val_dtype=vdt)
        dt = np.float64 if prec == "f64" else np.float32
        U = [u.astype(dt) for u in synth.random_factors(d, rank, seed=rank)]
        want = _reference(cidx, vals, U, None, 1e-10)
        # offset 0: aligned rows; offset 1: one element off a 16-byte boundary
        for off in (0, 1):
            dU = []
            for u in U:
                buf = torch.zeros(u.size + 1, dtype=torch.from_numpy(u).dtype, device="cuda")
                v = buf[off:off + u.size].view(u.shape)
                v.copy_(torch.from_numpy(u))
                dU.append(v)
            lam = torch.ones(rank, dtype=dU[0].dtype, device="cuda")
            got = ab.tt_logLikelihood(at, ab.KruskalModel([int(x) for x in d], rank, dU, lam))
            # FP64 products and sums of exact inputs (lambda is 1): at most ~1000 terms of relative error
            # N + R + 2 roundings each, far below 1e-12 of the sum of magnitudes
            scale = float((vals * 30).sum() + U[0].astype(np.float64).sum())
            assert abs(got - want) <= 1e-12 * scale, (nnz, off, got, want)
            # lambda holds mode 0's column sums: a sum of I positive terms in any order is within
            # (I - 1) roundings of the exact one, on both sides
            col, I = U[0].astype(np.float64).sum(0), U[0].shape[0]
            eps, got_lam = np.finfo(dt).eps, lam.cpu().numpy().astype(np.float64)
            assert np.allclose(got_lam, col, rtol=2 * np.finfo(np.float64).eps * I + eps, atol=0)
            # mode 0 comes back divided by them (one rounding of each)
            assert np.allclose(dU[0].cpu().numpy(), U[0] / got_lam, rtol=2 * eps, atol=0)
        at.destroy()
