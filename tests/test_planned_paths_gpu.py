"""The planned kernel's branches against a plain FP64 torch reference: ranks
without vector rows and misaligned factors (padded copies), modes read
through oidx, the Phi, tiles shared by several CTAs, outputs kept whole by
every CTA, the FP64 hot-row table, FP64 ranks of two chunks, and tile plans
whose indices span more than 22 bits.  Relative Frobenius error <= 1e-12
(FP64) and <= 1e-5 (FP32), the bounds of the other MTTKRP parity tests."""
import numpy as np
import pytest

import alto_b200 as ab
from alto_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOL = {"f64": 1e-12, "f32": 1e-5}
DT = {"f64": torch.float64, "f32": torch.float32}
EPS = 1e-10


def _tensor(dims, cidx, v, vdt):
    v = v.to({"f64": torch.float64, "f32": torch.float32, "u32": torch.int32}[vdt]).contiguous()
    return ab.create_alto_device(len(dims), np.array(dims, np.uint64), v.shape[0], cidx, v, 16, 0, val_dtype=vdt)


def _want(cidx, v, U, mode, phi):
    U = [u.double() for u in U]
    out = torch.zeros_like(U[mode])
    for o in range(0, v.shape[0], 1 << 20):
        s = slice(o, o + (1 << 20))
        p = torch.ones(cidx[0][s].shape[0], U[0].shape[1], dtype=torch.float64, device="cuda")
        for m in range(len(U)):
            if m != mode:
                p = p * U[m][cidx[m][s]]
        w = v[s].double()
        if phi:
            w = w / (U[mode][cidx[mode][s]] * p).sum(1).clamp(min=EPS)
        out.index_add_(0, cidx[mode][s], p * w[:, None])
    return out


def _factors(dims, rank, dt, seed, off=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    out = []
    for d in dims:
        buf = torch.empty(d * rank + 4, dtype=dt, device="cuda")
        u = buf[off:off + d * rank].view(d, rank)
        u.copy_(torch.rand(d, rank, dtype=dt, device="cuda", generator=g))
        out.append(u)
    return out


def _check(dims, cidx, v, rank, prec, vdt, off=0, modes=None, algo="auto", phi=(False, True)):
    at = _tensor(dims, cidx, v, vdt)
    vv = v.to(torch.int32) if vdt == "u32" else v.to(DT[prec])
    for mode in modes if modes is not None else range(len(dims)):
        for ph in phi:
            U = _factors(dims, rank, DT[prec], 3 * mode + rank, off)
            want = _want(cidx, vv, U, mode, ph)
            if ph:
                got = _factors(dims, rank, DT[prec], 1, off)[mode]
                ab.calculate_phi(at, mode, U, rank, got, EPS)
            else:
                # += semantics: on top of what the output holds
                want = want + U[mode].double()
                got = U[mode]
                ab.mttkrp_alto_par(mode, U, rank, at, algo=algo)
            err = float(torch.linalg.norm(got.double() - want) / torch.linalg.norm(want))
            assert err <= TOL[prec], (dims, v.shape[0], rank, prec, mode, "phi" if ph else "mttkrp", off, err)
    at.destroy()


@pytest.mark.parametrize("prec,vdt", [("f32", "f32"), ("f32", "u32"), ("f64", "f64"), ("f64", "u32")])
@pytest.mark.parametrize("dims", [(60, 50, 40), (30, 25, 20, 15), (14, 13, 12, 11, 10)])
@pytest.mark.parametrize("rank", [1, 2, 3, 5, 8, 25, 33, 64, 66, 100, 127])
def test_ranks_orders_types(dims, rank, prec, vdt):
    for nnz in (200, 5_001):
        cidx, v = synth.uniform_coo_torch(dims, nnz, nnz + rank, "cuda")
        _check(dims, cidx, torch.ceil(v * 9), rank, prec, vdt)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("rank,off", [(16, 1), (7, 1), (32, 3)])
def test_misaligned_factors(prec, rank, off):
    dims = (60, 50, 40)
    cidx, v = synth.uniform_coo_torch(dims, 4_000, 5, "cuda")
    _check(dims, cidx, v, rank, prec, prec, off=off)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("dims,rank", [((3000, 2500, 20), 16), ((4000, 30, 25, 3500), 8), ((9, 2000, 8, 7, 2600), 13),
                                       ((1 << 22, 1 << 21, 300), 4)])
def test_low_reuse_modes_through_oidx(dims, rank, prec):
    for nnz in (1, 33, 7_000):
        cidx, v = synth.uniform_coo_torch(dims, nnz, 9, "cuda")
        modes = [m for m in range(len(dims)) if nnz // dims[m] <= 4]
        _check(dims, cidx, v, rank, prec, prec, modes=modes, phi=(False,))


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_tile_shared_by_ctas_and_tile_edges(prec):
    dims = (300, 200, 100)
    for nnz in (1, 7, 1023, 1024, 1025, 40_000, 150_000):
        cidx, v = synth.uniform_coo_torch(dims, nnz, nnz, "cuda")
        _check(dims, cidx, v, 16, prec, prec)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("dims,rank", [((3000, 2000, 60), 16), ((900, 70, 800, 200), 25)])
def test_short_outputs_kept_whole(dims, rank, prec):
    cidx, v = synth.uniform_coo_torch(dims, 2_000_003, 2, "cuda")
    _check(dims, cidx, v, rank, prec, prec, modes=[m for m in range(len(dims)) if dims[m] <= 200])


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_hot_rows(prec):
    dims = (40_000, 30_000, 20_000)
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    n = 3_000_000
    # a few rows of every mode take most of the nonzeros
    cidx = torch.stack([(torch.rand(n, generator=g, device="cuda").pow(6) * d).long() for d in dims])
    v = 1.0 - torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    _check(dims, cidx, v, 32, prec, prec)


def test_plan_of_indices_past_22_bits():
    dims = (6_000_000, 50, 40)
    cidx, v = synth.uniform_coo_torch(dims, 3_000, 8, "cuda")
    cidx[0, :2] = torch.tensor([0, dims[0] - 1], device="cuda")
    _check(dims, cidx, v, 4, "f64", "f64", modes=[0], algo="tiled", phi=(False,))
