"""The build's sort over every width of high key words (none, 8, 32 and 64
bits), around its tile of 4096 keys and on digits that are all equal: the
encoding is bit-exact against the oracle.  And the library's memory pool
after a trim."""
import numpy as np
import pytest

import alto_b200 as ab
from alto_b200 import synth
from test_build_gpu import _check_against

pytestmark = pytest.mark.gpu

CASES = [
    ((1 << 21, 1 << 22, 1 << 21), 64),
    ((1 << 24, 1 << 24, 1 << 24), 72),
    ((1 << 25, 1 << 24, 1 << 24), 73),
    ((1 << 24, 1 << 24, 1 << 24, 1 << 24), 96),
    ((1 << 25, 1 << 24, 1 << 24, 1 << 24), 97),
    ((1 << 25, 1 << 25, 1 << 25, 1 << 25, 1 << 25), 125),
    ((5000, 3, 70, 1, 900), 32),
]


@pytest.mark.parametrize("dims,bits", CASES)
@pytest.mark.parametrize("nnz", [2, 4095, 4097, 13_000])
def test_sort_widths_and_tile_edges(oracle, dims, bits, nnz):
    dims_a, cidx, vals = synth.uniform_distinct(dims, nnz, seed=nnz + bits)
    lit = 64 if bits <= 64 else 128
    at = ab.create_alto(ab.SparseTensor.from_arrays(dims_a, cidx, vals), 7, lit)
    assert at.info()["alto_bits"] == bits
    _check_against(at.dump(), oracle.create(dims_a, cidx, vals, 7, lit).dump(), dims_a, nnz)


def test_sort_of_clustered_keys(oracle):
    """Most coordinates in one corner: high digits equal for nearly every key."""
    rng = np.random.default_rng(3)
    dims = np.array((1 << 24, 1 << 22, 1 << 20), np.uint64)
    cidx = np.stack([(rng.random(60_000) ** 12 * float(d)).astype(np.uint64) for d in dims])
    _, first = np.unique(cidx.T, axis=0, return_index=True)
    cidx = np.ascontiguousarray(cidx[:, np.sort(first)])
    vals = rng.random(cidx.shape[1])
    at = ab.create_alto(ab.SparseTensor.from_arrays(dims, cidx, vals), 16, 128)
    _check_against(at.dump(), oracle.create(dims, cidx, vals, 16, 128).dump(), dims, vals.shape[0])


def test_trim_returns_unused_memory():
    torch = pytest.importorskip("torch")
    cidx, v = synth.uniform_coo_torch((3000, 2000, 1000), 4_000_000, 1, "cuda")
    at = ab.create_alto_device(3, (3000, 2000, 1000), 4_000_000, cidx, v, 16, 0)
    at.destroy()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ab.trim_memory()
    # the build's buffers (at least keys, payloads and values of 4M nonzeros) were kept and came back
    assert torch.cuda.mem_get_info()[0] >= before + 4_000_000 * 20
