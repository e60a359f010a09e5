"""The build's sorts on both sides of the size up to which one block scans the
digit counts (128 tiles of 4096 keys), and well past it: keys, oidx and CR
bits bit-exact against the oracle."""
import pytest

import alto_b200 as ab
from alto_b200 import synth
from test_build_gpu import _check_against

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1 << 21, 1 << 20, 1 << 19), (1 << 24, 900, 1 << 23, 1 << 22)])
@pytest.mark.parametrize("nnz", [524_288, 524_289, 2_500_000])
def test_sort_past_the_one_block_scan(oracle, dims, nnz):
    dims_a, cidx, vals = synth.uniform_distinct(dims, nnz, seed=nnz)
    at = ab.create_alto(ab.SparseTensor.from_arrays(dims_a, cidx, vals), 9, 128)
    _check_against(at.dump(), oracle.create(dims_a, cidx, vals, 9, 128).dump(), dims_a, nnz)
