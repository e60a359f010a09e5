"""MTTKRP and Phi along short modes of small tensors, on both sides of the
rule that lets several CTAs share a tile (stretches of 2 to 128 records, 1 to
3000 rows), against the FP64 reference of the planned kernel's tests."""
import pytest

from alto_b200 import synth
from test_planned_paths_gpu import _check

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("rank", [2, 8, 16, 64, 100])
@pytest.mark.parametrize("dims", [(1, 20, 3000), (20, 20, 3000), (100, 40_000, 30), (50, 60, 7, 800)])
def test_short_modes(dims, rank, prec):
    for nnz in (1_025, 40_000, 100_000):
        cidx, v = synth.uniform_coo_torch(dims, nnz, nnz, "cuda")
        _check(dims, cidx, v, rank, prec, prec, phi=(False,))
        _check(dims, cidx, torch.ceil(v * 9), rank, prec, "u32", phi=(True,))
