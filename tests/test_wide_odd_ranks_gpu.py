"""FP64 MTTKRP and Phi at ranks above 64 that are no vector multiple, on both
sides of the rule that pads the factors or keeps the scalar rows, against the
FP64 reference of the planned kernel's tests."""
import pytest

from alto_b200 import synth
from test_planned_paths_gpu import _check

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rank", [65, 71, 73, 127])
@pytest.mark.parametrize("dims,nnz", [((300, 200, 100), 40_000), ((40_000, 25_000, 30), 90_000),
                                      ((6_000, 50, 40, 30, 20), 60_000), ((6_000, 50, 40, 30, 20), 20_000)])
def test_wide_odd_ranks(dims, nnz, rank):
    cidx, v = synth.uniform_coo_torch(dims, nnz, rank, "cuda")
    _check(dims, cidx, torch.ceil(v * 9), rank, "f64", "u32")
