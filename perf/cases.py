"""The calls that a user of alto_b200 makes, at the sizes of this repository's
configurations, tests and benchmark: MTTKRP along every mode, the CP-APR Phi,
the log-likelihood, the tensor build, CP-ALS, CP-APR and batched CP-ALS, each
through the package's public entry points.

A case is a dict:
  op       mttkrp | phi | loglik | build | cpals | cpapr | batch
  source   uniform (coordinates drawn uniformly), zipf (every mode's index
           Zipf(1.1), duplicates summed, log-normal values) or counts (Poisson
           counts of a Gamma(0.3, 1) Kruskal model, duplicates summed)
  dims     "4800000x1800000x1800000"
  draws    coordinates drawn (nonzeros for uniform; fewer after merging else)
  rank, dtype (f32 | f64: the model), vals (f32 | f64 | u32: stored values)
  iters, inner (solvers), tensors (batch)
"""
import math

import numpy as np
import torch

import alto_b200 as ab
from alto_b200 import synth

DEV = "cuda"
TORCH = {"f32": torch.float32, "f64": torch.float64}
EPS = 1e-10  # eps_div_zero of the CP-APR calls
NPRTN = 128  # the server's default partition count

CONFIG3 = "20000x10000x5000x200"
CONFIG2 = "4800000x1800000x1800000"


def listed():
    return [
        # the smallest calls: the package's own test and smoke tensor
        dict(name="mttkrp3_small_f64", op="mttkrp", source="uniform", dims="300x200x100", draws=40_000, rank=16,
             dtype="f64", vals="f64"),
        # the plain CP-ALS configuration's MTTKRP sweep
        dict(name="mttkrp3_uniform_f64", op="mttkrp", source="uniform", dims="1000x800x600", draws=1_000_000, rank=16,
             dtype="f64", vals="f64"),
        # the benchmark's headline: the large skewed tensor
        dict(name="mttkrp3_zipf_f32", op="mttkrp", source="zipf", dims=CONFIG2, draws=140_000_000, rank=32,
             dtype="f32", vals="f32"),
        # its FP64 companion, on a tensor that the solver's users decompose in FP64
        dict(name="mttkrp3_zipf_f64", op="mttkrp", source="zipf", dims=CONFIG2, draws=40_000_000, rank=32,
             dtype="f64", vals="f64"),
        # a sparse five-mode tensor of the batch configuration's ranges, alone: odd dimensions, modes of low
        # fiber reuse (read through oidx) beside modes of high reuse
        dict(name="mttkrp5_lowreuse_f32", op="mttkrp", source="uniform", dims="41203x17011x9973x2503x151",
             draws=150_001, rank=64, dtype="f32", vals="f32"),
        # counts with a rank that is no multiple of a vector
        dict(name="mttkrp4_counts_r25_f32", op="mttkrp", source="counts", dims=CONFIG3, draws=5_000_000, rank=25,
             dtype="f32", vals="u32"),
        # one Phi of the CP-APR configuration along each mode
        dict(name="phi4_counts_f32", op="phi", source="counts", dims=CONFIG3, draws=20_000_000, rank=16, dtype="f32",
             vals="u32"),
        # the log-likelihood check of an FP64 count model
        dict(name="loglik4_counts_f64", op="loglik", source="counts", dims=CONFIG3, draws=5_000_000, rank=16,
             dtype="f64", vals="u32"),
        # a tensor that has just arrived: build, then the first MTTKRP along every mode
        dict(name="build3_zipf_f32", op="build", source="zipf", dims=CONFIG2, draws=28_000_000, rank=32, dtype="f32",
             vals="f32"),
        # the plain CP-ALS configuration, whole
        dict(name="cpals3_uniform_f64", op="cpals", source="uniform", dims="1000x800x600", draws=1_000_000, rank=16,
             dtype="f64", vals="f64", iters=20),
        # CP-APR on counts of the CP-APR configuration's shape, whole, cut to a few outer iterations
        dict(name="cpapr4_counts_f32", op="cpapr", source="counts", dims=CONFIG3, draws=5_000_000, rank=16,
             dtype="f32", vals="u32", iters=4, inner=10),
        # batched CP-ALS of small independent tensors, whole
        dict(name="batch_cpals_f32", op="batch", source="counts", tensors=32, dtype="f32", vals="f32", iters=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_once(rng):
    op = rng.choice(["mttkrp"] * 6 + ["phi"] * 2 + ["loglik"] * 2 + ["build"] * 2 + ["cpals"] * 2 + ["cpapr"] + ["batch"])
    if op == "batch":
        return dict(op=op, source="counts", tensors=rng.randint(12, 40), dtype="f32", vals="f32",
                    iters=rng.randint(3, 4))
    rank = rng.choice([8, 16, 32, 64]) if rng.random() < 0.6 else rng.randint(3, 80)
    source = {"mttkrp": rng.choice(["uniform", "zipf", "counts"]), "phi": "counts", "loglik": "counts",
              "build": rng.choice(["uniform", "zipf", "counts"]), "cpals": rng.choice(["uniform", "counts"]),
              "cpapr": "counts"}[op]
    dtype = rng.choice(["f32", "f32", "f64"])
    if op == "cpals" and source == "uniform":
        dtype = "f64"
    if source == "uniform":
        dims = [_log_int(rng, 100, 50_000) for _ in range(rng.choice([3, 4, 5]))]
        draws = _log_int(rng, 10_000, 2_000_000 if op == "cpals" else 5_000_000)
        vals = dtype
    elif source == "zipf":
        dims = [_log_int(rng, 300_000, 5_000_000) for _ in range(3)]
        draws = _log_int(rng, 500_000, 30_000_000 if op == "build" else 100_000_000)
        vals = dtype
    else:
        dims = [_log_int(rng, lo, hi) for lo, hi in ((5_000, 50_000), (2_000, 20_000), (1_000, 10_000), (100, 500))]
        rng.shuffle(dims)
        draws = _log_int(rng, 50_000, {"cpals": 2_000_000, "cpapr": 3_000_000}.get(op, 20_000_000))
        vals = dtype if op == "cpals" else "u32"
    case = dict(op=op, source=source, dims="x".join(map(str, dims)), draws=draws, rank=rank, dtype=dtype, vals=vals)
    if op == "cpals":
        case["iters"] = rng.randint(3, 10)
    if op == "cpapr":
        case["iters"], case["inner"] = rng.randint(2, 4), rng.randint(2, 10)
    return case


def draw(rng):
    most = work(listed()[2])
    while True:
        case = _draw_once(rng)
        w = work(case)
        if w["bytes"] <= most["bytes"] and w["flops"] <= most["flops"]:
            return case


# ------------------------------------------------------------------ inputs

def _dims(case):
    return [int(d) for d in case["dims"].split("x")]


def _coo(case, seed):
    """(dims, cidx int64 (modes, nnz), values of the stored type), on the GPU."""
    dims, draws = _dims(case), case["draws"]
    if case["source"] == "uniform":
        cidx, v = synth.uniform_coo_torch(dims, draws, seed, DEV)
    elif case["source"] == "zipf":
        cidx, v = _zipf(dims, draws, 1.1, seed)
    else:
        cidx, v = synth.poisson_kruskal_torch(dims, 10, draws, seed, DEV)
    if case["vals"] != "u32":
        v = v.to(TORCH[case["vals"]])
    return dims, cidx.contiguous(), v.contiguous()


def _zipf(dims, draws, s, seed):
    """Three-mode Zipf(s) coordinates in lexicographic order, repeated ones merged by summing log-normal values
    (synth.zipf_tensor_torch's distribution).  The values are whole multiples of 2^-20, so their sums do not depend on
    the order in which they are added."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    idx = []
    for d in dims:
        cdf = torch.cumsum(torch.arange(1, d + 1, dtype=torch.float64, device=DEV).pow_(-s), 0)
        cdf /= cdf[-1].clone()
        idx.append(torch.searchsorted(cdf, torch.rand(draws, dtype=torch.float64, device=DEV, generator=g), right=True)
                   .clamp_(max=d - 1))
    v = torch.exp(torch.randn(draws, dtype=torch.float64, device=DEV, generator=g))
    v.mul_(1 << 20).round_().mul_(2.0**-20)
    low = idx[1].mul_(dims[2]).add_(idx[2])
    order = torch.sort(low, stable=True).indices
    order = order[torch.sort(idx[0][order], stable=True).indices]
    i0, low, v = idx[0][order], low[order], v[order]
    new = torch.ones(draws, dtype=torch.bool, device=DEV)
    new[1:] = (i0[1:] != i0[:-1]) | (low[1:] != low[:-1])
    seg = torch.cumsum(new, 0).sub_(1)
    v = torch.zeros(int(seg[-1]) + 1, dtype=torch.float64, device=DEV).index_add_(0, seg, v)
    i0, low = i0[new], low[new]
    return torch.stack([i0, low // dims[2], low % dims[2]]), v


def _factors(case, dims, rank, seed):
    """Uniform (0, 1) factors in the model's type."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1009 + 17)
    return [torch.rand(d, rank, dtype=TORCH[case["dtype"]], device=DEV, generator=g) for d in dims]


def _batch_shapes(case):
    # the shapes are the case's own (order 3 to 5, dims 100 to 50,000, 10,000 to 2,000,000 draws, rank 8 to 32); the
    # coordinates and counts are the seed's.  Rank 64 on these would be nearly singular in FP32: its lambdas differ
    # from run to run.
    return synth.batch_shapes(case["tensors"], seed=case["tensors"], ranks=(8, 16, 32))


def _tensor(dims, cidx, v, vals):
    return ab.create_alto_device(len(dims), np.array(dims, np.uint64), v.shape[0], cidx, v, NPRTN, 0, val_dtype=vals)


def _carve(shapes, dtype):
    """One buffer and its views of the given shapes, each on a 256-byte boundary."""
    offs, n = [], 0
    for s in shapes:
        offs.append(n)
        n += (math.prod(s) + 63) // 64 * 64
    flat = torch.zeros(max(n, 1), dtype=dtype, device=DEV)
    return flat, [flat[o:o + math.prod(s)].view(s) for o, s in zip(offs, shapes)]


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        return _prepare_batch(case, seed)
    dims, cidx, v = _coo(case, seed)
    rank = case["rank"]
    st = {"op": op, "case": case, "dims": dims, "rank": rank}
    U = _factors(case, dims, rank, seed)
    if op == "build":
        st["cidx"], st["v"] = cidx, v
    else:
        st["at"] = _tensor(dims, cidx, v, case["vals"])
        del cidx, v
    if op in ("mttkrp", "build"):
        st["U"], st["out"] = U, [torch.zeros_like(u) for u in U]
    elif op == "phi":
        st["U"], st["out"] = U, [torch.zeros_like(u) for u in U]
    else:
        # the solvers work in place: the initial model is kept and copied in before each pass
        dt = TORCH[case["dtype"]]
        st["init"], views = _carve([(d, rank) for d in dims] + [(rank,)], dt)
        for x, y in zip(views, U + [torch.ones(rank, dtype=dt, device=DEV)]):
            x.copy_(y)
        st["flat"], views = _carve([(d, rank) for d in dims] + [(rank,)], dt)
        st["M"] = ab.KruskalModel(dims, rank, views[:-1], views[-1])
    torch.cuda.synchronize()
    return st


def _prepare_batch(case, seed):
    dt = TORCH[case["dtype"]]
    tensors, shapes, init = [], [], []
    for k, (dims, nnz, rank) in enumerate(_batch_shapes(case)):
        cidx, v = synth.poisson_kruskal_torch(dims, 32, nnz, seed * 7919 + k, DEV)
        tensors.append(_tensor(dims, cidx, v.to(dt), case["vals"]))
        shapes += [(d, rank) for d in dims] + [(rank,)]
        init += _factors(case, dims, rank, seed * 131 + k) + [torch.ones(rank, dtype=dt, device=DEV)]
    keep, views = _carve(shapes, dt)
    for x, y in zip(views, init):
        x.copy_(y)
    flat, views = _carve(shapes, dt)
    models, at = [], 0
    for dims, nnz, rank in _batch_shapes(case):
        models.append(ab.KruskalModel(list(dims), rank, views[at:at + len(dims)], views[at + len(dims)]))
        at += len(dims) + 1
    batch = ab.BatchCPD(tensors, models, fit_capacity=case["iters"])
    torch.cuda.synchronize()
    return {"op": "batch", "case": case, "batch": batch, "init": keep, "flat": flat}


# -------------------------------------------------------------------- a pass

def _sweep(st, at):
    U, out = st["U"], st["out"]
    for n in range(len(out)):
        ab.mttkrp_alto_par(n, [out[m] if m == n else U[m] for m in range(len(U))], st["rank"], at, accumulate=False)
    return out


def run(st):
    op, case = st["op"], st["case"]
    if op == "mttkrp":
        return _sweep(st, st["at"])
    if op == "build":
        at = _tensor(st["dims"], st["cidx"], st["v"], case["vals"])
        out = _sweep(st, at)
        at.destroy()
        return out
    if op == "phi":
        for n in range(len(st["U"])):
            ab.calculate_phi(st["at"], n, st["U"], st["rank"], st["out"][n], EPS)
        return st["out"]
    st["flat"].copy_(st["init"])
    if op == "batch":
        fits, iters = st["batch"].solve(case["iters"], 0.0)
        return {"fits": fits, "iters": iters, "models": st["flat"]}
    M = st["M"]
    if op == "loglik":
        return {"loglik": ab.tt_logLikelihood(st["at"], M, EPS), "U0": M.U[0], "lam": M.lam}
    if op == "cpals":
        fits = ab.cpd_alto(st["at"], M, case["iters"], 0.0)
        return {"fits": fits, "U": M.U, "lam": M.lam}
    s = ab.cp_apr_alto(st["at"], M, case["iters"], case["inner"], 1e-5, EPS)
    return {"loglik": s["loglik"], "fit": s["fit"], "kkt": s["kkt"], "outer": s["outer"], "inner": s["inner"], "U": M.U,
            "lam": M.lam}


# ---------------------------------------------------------------------- work

def _nnz(case):
    """Nonzeros after merging, as a share of the draws that holds at these sizes."""
    return case["draws"] * {"uniform": 1.0, "zipf": 0.72, "counts": 0.95}[case["source"]]


def _sweep_work(nnz, dims, rank, fsz, vsz):
    """MTTKRP along every mode: key and value of each nonzero, the other modes' factors in, one factor out."""
    n = len(dims)
    return n * (nnz * (8 + vsz) + sum(dims) * rank * fsz), n * nnz * rank * n


def work(case):
    op = case["op"]
    fsz = 8 if case["dtype"] == "f64" else 4
    vsz = 8 if case["vals"] == "f64" else 4
    if op == "batch":
        b = f = 0
        for dims, nnz, rank in _batch_shapes(case):
            sb, sf = _sweep_work(nnz, dims, rank, fsz, vsz)
            b += case["iters"] * sb
            f += case["iters"] * (sf + sum(dims) * rank * rank * 4)
        return {"bytes": b, "flops": f}
    dims, rank, nnz = _dims(case), case["rank"], _nnz(case)
    n = len(dims)
    b, f = _sweep_work(nnz, dims, rank, fsz, vsz)
    if op == "build":  # coordinates and values in, the encoding out, then the sweep
        return {"bytes": b + nnz * (8 * n + vsz + 8 + vsz), "flops": f}
    if op == "phi":  # the target's factor is read too
        return {"bytes": b + sum(dims) * rank * fsz, "flops": f + n * nnz * rank * 3}
    if op == "loglik":
        return {"bytes": nnz * (8 + vsz) + (sum(dims) + 2 * dims[0]) * rank * fsz, "flops": nnz * rank * n}
    if op == "cpals":
        it = case["iters"]
        return {"bytes": it * (b + 2 * sum(dims) * rank * fsz), "flops": it * (f + sum(dims) * rank * rank * 4)}
    if op == "cpapr":  # one Phi of every mode per inner iteration, B updated in place
        it = case["iters"] * case["inner"]
        return {"bytes": it * (b + 2 * sum(dims) * rank * fsz), "flops": it * (f + n * nnz * rank * 3)}
    return {"bytes": b, "flops": f}


# --------------------------------------------------------------------- exact

CHUNK = 1 << 21


def _krp(cidx, U, mode, s):
    """Products of the other modes' rows of the nonzeros in slice s."""
    p = None
    for m, u in enumerate(U):
        if m != mode:
            r = u[cidx[m][s]]
            p = r if p is None else p.mul_(r)
    return p


def _mttkrp64(cidx, v, U, mode):
    out = torch.zeros_like(U[mode])
    for o in range(0, v.shape[0], CHUNK):
        s = slice(o, o + CHUNK)
        out.index_add_(0, cidx[mode][s], _krp(cidx, U, mode, s).mul_(v[s, None]))
    return out


def _phi64(cidx, v, U, mode):
    out = torch.zeros_like(U[mode])
    for o in range(0, v.shape[0], CHUNK):
        s = slice(o, o + CHUNK)
        p = _krp(cidx, U, mode, s)
        d = (U[mode][cidx[mode][s]] * p).sum(1).clamp_(min=EPS)
        out.index_add_(0, cidx[mode][s], p.mul_((v[s] / d)[:, None]))
    return out


def _loglik64(cidx, v, U, lam):
    """tt_logLikelihood in place: lambda into mode 0, the sum, mode 0 normalised again."""
    U[0].mul_(lam)
    ll = 0.0
    for o in range(0, v.shape[0], CHUNK):
        s = slice(o, o + CHUNK)
        ll += float((v[s] * _krp(cidx, U, -1, s).sum(1).clamp_(min=EPS).log()).sum())
    ll -= float(U[0].sum())
    lam.copy_(U[0].abs().sum(0))
    U[0].div_(lam)
    return ll


def _fit64(U, lam, M, xx):
    """1 - |X - model| / |X| with the last mode's MTTKRP M."""
    g = torch.outer(lam, lam)
    for u in U:
        g = g * (u.t() @ u)
    res = float(xx + g.sum().abs() - 2.0 * ((U[-1] * M).sum(0) * lam).sum())
    return 1.0 - (math.sqrt(res) if res > 0 else res) / math.sqrt(float(xx))


def _cpals64(cidx, v, U, iters):
    n, xx, fits = len(U), (v * v).sum(), []
    lam = torch.ones(U[0].shape[1], dtype=torch.float64, device=DEV)
    for it in range(iters):
        for j in range(n):
            M = _mttkrp64(cidx, v, U, j)
            V = torch.ones(len(lam), len(lam), dtype=torch.float64, device=DEV)
            for m in range(n):
                if m != j:
                    V = V * (U[m].t() @ U[m])
            L, bad = torch.linalg.cholesky_ex(V)
            if int(bad):
                return None  # the pseudo-inverse's cut-off is the solver's own
            Y = torch.cholesky_solve(M.t().contiguous(), L).t().contiguous()
            lam = Y.square().sum(0).sqrt() if it == 0 else Y.max(0).values.clamp(min=1.0)
            U[j] = Y / lam
        fits.append(_fit64(U, lam, M, xx))
    return np.array(fits), U, lam


def _cpapr64(cidx, v, U, outer, inner, eps=1e-5, kappa_tol=1e-10, kappa=1e-2):
    n = len(U)
    lam = torch.ones(U[0].shape[1], dtype=torch.float64, device=DEV)
    Phi, kkts, kmode = [None] * n, [], [0.0] * n

    def normalise(j):
        c = U[j].abs().sum(0)
        U[j].div_(c)
        lam.mul_(c)

    for j in range(n):
        normalise(j)
    done = outer
    for it in range(outer):
        for j in range(n):
            if it:
                U[j] = torch.where((U[j] < kappa_tol) & (Phi[j] > 1.0), U[j] + kappa, U[j])
            U[j].mul_(lam)
            lam.fill_(1.0)
            for _ in range(inner):
                Phi[j] = _phi64(cidx, v, U, j)
                kmode[j] = float(torch.minimum(U[j], 1.0 - Phi[j]).abs().max())
                if kmode[j] < eps:
                    break
                U[j].mul_(Phi[j])
            normalise(j)
        kkts.append(max(kmode))
        if it and abs(kkts[it] - kkts[it - 1]) <= eps * eps:
            done = it
            break
    ll = _loglik64(cidx, v, U, lam)
    fit = _fit64(U, lam, _mttkrp64(cidx, v, U, n - 1), (v * v).sum())
    return dict(loglik=ll, fit=fit, kkt=kkts[max(done - 1, 0)], outer=None, inner=None, U=U, lam=lam)


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        return None  # dozens of solves, some with nearly singular normal equations
    dims, cidx, v = _coo(case, seed)
    v = v.double()
    U = [u.double() for u in _factors(case, dims, case["rank"], seed)]
    if op in ("mttkrp", "build"):
        return [_mttkrp64(cidx, v, U, n) for n in range(len(dims))]
    if op == "phi":
        return [_phi64(cidx, v, U, n) for n in range(len(dims))]
    if op == "loglik":
        lam = torch.ones(case["rank"], dtype=torch.float64, device=DEV)
        ll = _loglik64(cidx, v, U, lam)
        return {"loglik": ll, "U0": U[0], "lam": lam}
    if op == "cpals":
        got = _cpals64(cidx, v, U, case["iters"])
        return None if got is None else {"fits": got[0], "U": got[1], "lam": got[2]}
    return _cpapr64(cidx, v, U, case["iters"], case["inner"])
