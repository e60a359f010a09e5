"""The device bytes that a handle reports hold the buffers it keeps between
calls, and its destruction gives them back."""
import numpy as np
import pytest

import alto_b200 as ab
from alto_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_handle_reports_its_buffers():
    dims, rank, nnz = (30_000, 20_000, 10_000), 25, 400_000
    cidx, v = synth.uniform_coo_torch(dims, nnz, 1, "cuda")
    at = ab.create_alto_device(3, np.array(dims, np.uint64), nnz, cidx, v.float(), 16, 0, val_dtype="f32")
    before = at.info()["device_bytes"]
    assert before >= nnz * 12
    U = [torch.rand(d, rank, device="cuda") for d in dims]
    ab.mttkrp_alto_par(0, U, rank, at)
    torch.cuda.synchronize()
    assert at.info()["device_bytes"] >= before + sum(dims) * 28 * 4  # rows of 25 floats padded to 28
    held = at.info()["device_bytes"]
    ab.mttkrp_alto_par(0, U, rank, at)
    assert at.info()["device_bytes"] == held
    at.destroy()
