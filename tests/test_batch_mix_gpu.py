"""Batched CP-ALS where the dense update runs its rank classes side by side
(fused classes up to 64 beside ranks above), and batches with more tensors of
one class than the tile lookup keeps in shared memory: every tensor must give
what a separate solve gives (FP64: fits within 1e-9, factors within 1e-7, the
tolerances of the other batched tests)."""
import numpy as np
import pytest

import alto_b200 as ab
from alto_b200 import synth
from conftest import rel_fro
from test_batch_gpu import _model

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _compare(items, iters, check, use_graph):
    models = [_model(dims, rank, 7 + k, np.float64) for k, (dims, at, rank) in enumerate(items)]
    b = ab.BatchCPD([at for _, at, _ in items], models, fit_capacity=iters)
    fits, its = b.solve(iters, 0.0, use_graph=use_graph)
    assert (its == iters).all()
    for k in check:
        dims, at, rank = items[k]
        M = _model(dims, rank, 7 + k, np.float64)
        want = ab.cpd_alto(at, M, iters, 0.0)
        assert np.allclose(fits[k], want, rtol=0, atol=1e-9), (k, rank, fits[k], want)
        for u, v in zip(models[k].U, M.U):
            assert rel_fro(u.cpu().numpy(), v.cpu().numpy()) < 1e-7, (k, rank)
        assert rel_fro(models[k].lam.cpu().numpy(), M.lam.cpu().numpy()) < 1e-7
    b.close()


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("ranks", [(5,), (70,), (8, 16), (8, 30, 100), (4, 12, 20, 40, 64, 70, 96)])
def test_rank_classes_side_by_side(ranks, use_graph):
    items = []
    for k, r in enumerate(ranks):
        for dims in ((150, 120, 110), (130, 100, 110, 105)):
            d, cidx, vals = synth.uniform_distinct(dims, 20_000, seed=r + len(dims))
            items.append((d, ab.create_alto(ab.SparseTensor.from_arrays(d, cidx, vals), 8, 0), r))
    _compare(items, 3, range(len(items)), use_graph)


def test_more_tensors_than_the_tile_lookup_holds():
    items = []
    for k in range(530):
        d, cidx, vals = synth.uniform_distinct((12, 11, 10), 300, seed=k)
        items.append((d, ab.create_alto(ab.SparseTensor.from_arrays(d, cidx, vals), 4, 0), 4))
    _compare(items, 2, (0, 1, 255, 511, 512, 513, 529), True)
