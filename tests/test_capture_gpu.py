"""MTTKRP and Phi recorded in CUDA graphs: what a graph's calls use stays
theirs when later calls on the handle need larger buffers, and graphs of one
handle replayed side by side do not disturb each other."""
import numpy as np
import pytest

import alto_b200 as ab
from alto_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOL = {"f64": 1e-12, "f32": 1e-5}  # the parity tests' bounds
DT = {"f64": torch.float64, "f32": torch.float32}


def _sweep(at, U, rank, out, phi, stream):
    for n in range(len(U)):
        if phi:
            ab.calculate_phi(at, n, U, rank, out[n], stream=stream)
        else:
            ab.mttkrp_alto_par(n, [out[m] if m == n else U[m] for m in range(len(U))], rank, at, accumulate=False,
                               stream=stream)


def _factors(dims, rank, dt, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return [torch.rand(d, rank, dtype=dt, device="cuda", generator=g) for d in dims]


def _record(at, U, rank, phi):
    out = [torch.full_like(u, 7) for u in U]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    side = torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side, capture_error_mode="thread_local"):
        _sweep(at, U, rank, out, phi, side)
    return graph, out


def _near(got, want, prec):
    for a, b in zip(got, want):
        assert float(torch.linalg.norm(a.double() - b.double()) / torch.linalg.norm(b.double())) <= TOL[prec]


def _tensor(dims, nnz, prec, seed):
    cidx, v = synth.uniform_coo_torch(dims, nnz, seed, "cuda")
    return ab.create_alto_device(len(dims), np.array(dims, np.uint64), nnz, cidx, v.to(DT[prec]), 16, 0, val_dtype=prec)


@pytest.mark.parametrize("phi", [False, True])
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("rank", [4, 25])
def test_graph_outlives_growth_of_the_handle(rank, prec, phi):
    dims = (900, 700, 60)
    at = _tensor(dims, 300_000, prec, rank)
    U = _factors(dims, rank, DT[prec], 1)
    want = [torch.zeros_like(u) for u in U]
    _sweep(at, U, rank, want, phi, torch.cuda.current_stream())
    graph, out = _record(at, U, rank, phi)
    for r in (64, 127, 128):  # larger accumulators and padded copies than the graph's call
        V = _factors(dims, r, DT[prec], r)
        for p in (False, True):
            _sweep(at, V, r, [torch.zeros_like(u) for u in V], p, torch.cuda.current_stream())
    others = [_tensor(dims, 400_000, prec, s) for s in range(3)]  # what was given back is in use elsewhere
    want2 = [o.dump() for o in others]
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    _near(out, want, prec)
    for o, w in zip(others, want2):
        d = o.dump()
        assert np.array_equal(d["idx"], w["idx"]) and np.array_equal(d["vals"], w["vals"])
    # the handle still answers eager calls
    again = [torch.zeros_like(u) for u in U]
    _sweep(at, U, rank, again, phi, torch.cuda.current_stream())
    _near(again, want, prec)
    del graph
    torch.cuda.synchronize()
    at.destroy()


@pytest.mark.parametrize("phi", [False, True])
@pytest.mark.parametrize("rank", [16, 25])
def test_fp64_graphs_of_one_handle_side_by_side(rank, phi):
    dims = (20_000, 15_000, 90)
    at = _tensor(dims, 3_000_000, "f64", 2)
    runs = []
    for seed in (1, 2):
        U = _factors(dims, rank, torch.float64, seed)
        want = [torch.zeros_like(u) for u in U]
        _sweep(at, U, rank, want, phi, torch.cuda.current_stream())
        runs.append((U, want) + _record(at, U, rank, phi))
    streams = [torch.cuda.Stream() for _ in runs]
    torch.cuda.synchronize()
    for _ in range(5):
        for (U, want, graph, out), st in zip(runs, streams):
            with torch.cuda.stream(st):
                graph.replay()
    torch.cuda.synchronize()
    for U, want, graph, out in runs:
        _near(out, want, "f64")
    del runs
    torch.cuda.synchronize()
    at.destroy()
