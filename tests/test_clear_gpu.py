"""The clearing of an MTTKRP's output beside the kernel that follows it: on
both sides of the sizes where it is a kernel of its own (32 MB of gathers, a
16 MB output) and where the next kernel starts early (a 512 KB output, two
tiles an SM), every element of the output is replaced, call after call."""
import numpy as np
import pytest

import alto_b200 as ab
from alto_b200 import synth
from test_planned_paths_gpu import DT, TOL, _factors, _want

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("dims,nnz,rank", [
    ((300, 200, 100), 40_000, 16),                    # memset
    ((1_000, 800, 600), 1_000_000, 32),               # small outputs
    ((20_000, 4_100, 2_040), 700_000, 32),            # 512 KB lies between the modes
    ((41_203, 17_011, 9_973, 2_503, 151), 150_001, 64),  # shared tiles
    ((70_000, 30_000, 20), 600_000, 64),              # 16 MB lies between the modes
])
def test_outputs_are_replaced(dims, nnz, rank, prec):
    cidx, v = synth.uniform_coo_torch(dims, nnz, nnz, "cuda")
    v = v.to(DT[prec])
    at = ab.create_alto_device(len(dims), np.array(dims, np.uint64), nnz, cidx, v, 16, 0, val_dtype=prec)
    U = _factors(dims, rank, DT[prec], 5)
    out = [torch.full_like(u, 1e6) for u in U]
    for call in range(3):  # the modes one after another on one stream, twice over their own results
        for n in range(len(dims)):
            ab.mttkrp_alto_par(n, [out[m] if m == n else U[m] for m in range(len(dims))], rank, at, accumulate=False)
    for n in range(len(dims)):
        want = _want(cidx, v, U, n, False)
        assert float(torch.linalg.norm(out[n].double() - want) / torch.linalg.norm(want)) <= TOL[prec], n
    at.destroy()
