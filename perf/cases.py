"""Timed cases of the solver: whole least-squares solves through the public entry points.

Every case is one call a user makes: a sparse solve (device buffers or host
arrays), a dense solve with any of the three dense solvers, or a batch of small
sparse problems.  Inputs follow synthetic.py's distributions, made on the GPU.
Solves ask for a tight LSQR tolerance, so x is the least-squares solution
itself and not a point on the way to it.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "ski-lls_gb300"))
import skills_gb300 as skl  # noqa: E402

IT_TOL = 1e-12


def _sparse(name, n, d, per_col, gamma, k, **kw):
    c = dict(name=name, kind="sparse", n=n, d=d, per_col=per_col, gamma=gamma, k=k, via="device",
             precision="mixed", profile="uniform", scale_exp=0.0, n_dep=0, noise=1e-3)
    c.update(kw)
    return c


def _dense(name, n, d, solver, kappa_exp, gamma, k, **kw):
    c = dict(name=name, kind="dense", n=n, d=d, solver=solver, kappa_exp=kappa_exp, gamma=gamma,
             k=k, precision="mixed", noise=1e-4)
    c.update(kw)
    return c


def listed():
    return [
        # a small regression from host arrays: latency and launches only
        _sparse("sparse_2000x60_host", 2000, 60, 100, 1.7, 2, via="host"),
        # uniform 1 % sparse matrix, the ordinary size
        _sparse("sparse_20000x1000", 20000, 1000, 200, 1.7, 2),
        # odd sizes, badly scaled columns, the solver's default sketch (gamma 1.1, k 3)
        _sparse("sparse_31013x1507", 31013, 1507, 311, 1.1, 3, scale_exp=4.0),
        # large 1 % sparse matrix with badly scaled columns, full rank
        _sparse("sparse_120000x5000", 120000, 5000, 1200, 1.7, 2, scale_exp=4.0),
        # the same with column scales up to 1e8 and 50 dependent columns: x is not
        # unique, the fitted values A x and the rank are what such a user reads
        _sparse("sparse_rankdef_120000x5000", 120000, 5000, 1200, 1.7, 2, scale_exp=8.0, n_dep=50,
                noise=1e-6),
        # power-law column lengths, the largest sparse problem
        _sparse("sparse_zipf_1000000x10000", 1000000, 10000, 1000, 1.5, 3, profile="zipf",
                noise=-1.0),
        # the all-FP64 option
        _sparse("sparse_fp64_20000x1000", 20000, 1000, 200, 1.7, 2, precision="fp64"),
        # a small dense regression with odd sizes
        _dense("dense_5003x301", 5003, 301, "hashing", 2.0, 1.7, 1),
        # unpivoted dense solver, ordinary size
        _dense("dense_nocpqr_12007x1201", 12007, 1201, "nocpqr", 3.0, 1.7, 1),
        # ill-conditioned dense problem, pivoted sketch QR
        _dense("dense_40000x4000", 40000, 4000, "hashing", 4.0, 1.7, 1),
        # Blendenpik at its driver's gamma
        _dense("dense_blendenpik_40000x4000", 40000, 4000, "blendenpik", 3.0, 2.2, 1),
        # many small host problems in one call
        dict(name="batched_64", kind="batched", count=64, shapes=2024, d_min=50, d_max=500,
             n_max=50000, gamma=1.7, k=2),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what = rng.choice(["sparse", "sparse", "sparse", "rankdef", "zipf", "fp64", "dense", "dense",
                       "batched"])
    if what == "batched":
        d_max = rng.randint(100, 500)
        return dict(kind="batched", count=rng.randint(8, 64), shapes=rng.randrange(1 << 30),
                    d_min=50, d_max=d_max, n_max=rng.randint(10000, 50000), gamma=rng.choice([1.4, 1.7]), k=2)
    if what == "dense":
        d = _log_int(rng, 50, 4000)
        n = min(40000, _log_int(rng, 10 * d, 60 * d))
        solver = rng.choice(["hashing", "hashing", "nocpqr", "blendenpik"])
        # the unpivoted solvers start LSQR from 0: beyond 1e3 their x keeps fewer digits
        c = _dense("", n, d, solver, rng.uniform(0.0, 4.0 if solver == "hashing" else 3.0),
                   2.2 if solver == "blendenpik" else rng.choice([1.4, 1.7]), 1)
        del c["name"]
        return c
    k = rng.choice([2, 3])
    gamma = rng.choice([1.1, 1.4, 1.7])
    if what == "zipf":
        d = _log_int(rng, 1000, 8000)
        n = _log_int(rng, 40 * d, 100 * d)
        c = _sparse("", n, d, rng.randint(100, 1000), rng.choice([1.4, 1.5, 1.7]), k,
                    profile="zipf", noise=-1.0)
    elif what == "rankdef":
        d = _log_int(rng, 500, 5000)
        n = _log_int(rng, 20 * d, 30 * d)
        c = _sparse("", n, d, max(8, n // 100), rng.choice([1.4, 1.7]), k, scale_exp=8.0,
                    n_dep=rng.randint(1, max(1, d // 100)), noise=1e-6)
    else:
        d = _log_int(rng, 50, 1500 if what == "fp64" else 6000)
        n = _log_int(rng, max(2000, 20 * d), max(2000, 50 * d))
        per_col = max(8, min(int(round(n * rng.uniform(0.004, 0.02))), 10000000 // d))
        c = _sparse("", n, d, per_col, gamma, k, scale_exp=rng.choice([0.0, 4.0]),
                    precision="fp64" if what == "fp64" else "mixed",
                    via="host" if d < 1000 and rng.random() < 0.3 else "device")
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs --
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _normal(g, *size):
    return torch.randn(*size, generator=g, device="cuda", dtype=torch.float64)


def _csc_matrix(c, seed):
    """(p, i, x): int64 column pointers, sorted int64 rows, FP64 values, on the GPU."""
    n, d = c["n"], c["d"]
    g = _generator(seed)
    if c["profile"] == "zipf":
        cap = max(20, n // 50)
        raw = np.minimum(np.random.default_rng(seed).zipf(1.2, size=d), cap).astype(np.float64)
        counts = np.round(raw * (c["per_col"] * d / raw.sum())).astype(np.int64)
        # at least 8 entries: shorter columns coincide now and then, and x is then not unique
        counts = torch.from_numpy(np.clip(counts, 8, cap)).cuda()
    else:
        counts = torch.full((d,), c["per_col"], dtype=torch.int64, device="cuda")
    cols = torch.repeat_interleave(torch.arange(d, device="cuda"), counts)
    rows = torch.randint(0, n, (cols.numel(),), generator=g, device="cuda")
    keys = torch.unique(cols * n + rows)          # sorted by column, then row
    vals = _normal(g, keys.numel())
    if c["scale_exp"] > 0:
        scale = 10.0 ** (c["scale_exp"] * torch.rand(d, generator=g, device="cuda",
                                                     dtype=torch.float64))
        vals = vals * scale[keys // n]
    if c["n_dep"]:
        # column dep[t] becomes a[t] * column p[t] + b[t] * column q[t]
        t = c["n_dep"]
        order = torch.randperm(d, generator=g, device="cuda")
        dep, kept = order[:t], order[t:]
        pq = kept[torch.randint(0, d - t, (2, t), generator=g, device="cuda")]
        ab = _normal(g, 2, t)
        is_dep = torch.zeros(d, dtype=torch.bool, device="cuda")
        is_dep[dep] = True
        keep = ~is_dep[keys // n]
        keys, vals = keys[keep], vals[keep]
        col = keys // n
        more_k, more_v = [keys], [vals]
        for s in range(t):
            for w in range(2):
                at = col == pq[w, s]
                more_k.append(dep[s] * n + keys[at] % n)
                more_v.append(ab[w, s] * vals[at])
        keys, inv = torch.unique(torch.cat(more_k), return_inverse=True)
        vals = torch.zeros(keys.numel(), dtype=torch.float64, device="cuda").index_add_(
            0, inv, torch.cat(more_v))
    p = torch.zeros(d + 1, dtype=torch.int64, device="cuda")
    p[1:] = torch.cumsum(torch.bincount(keys // n, minlength=d), 0)
    return p, (keys % n).contiguous(), vals.contiguous()


def _csr(c, p, i, x):
    cols = torch.repeat_interleave(torch.arange(c["d"], device="cuda"), p[1:] - p[:-1])
    order = torch.argsort(i * c["d"] + cols)
    rp = torch.zeros(c["n"] + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(i, minlength=c["n"]), 0)
    return torch.sparse_csr_tensor(rp, cols[order], x[order], size=(c["n"], c["d"]))


def _sparse_inputs(c, seed):
    p, i, x = _csc_matrix(c, seed)
    A = _csr(c, p, i, x)
    g = _generator(seed + 1)
    if c["noise"] < 0:                            # b with no relation to A
        b = _normal(g, c["n"])
    else:
        b = A @ _normal(g, c["d"]) + c["noise"] * _normal(g, c["n"])
    return p, i, x, b, A


def _hartley_rows(X):
    F = torch.fft.fft(X, dim=1)
    return (F.real - F.imag) / math.sqrt(X.shape[1])


def _dense_inputs(c, seed):
    """A = G diag(logspace(0, -kappa_exp)) Q, Gaussian G / sqrt(n) and orthogonal
    Q, stored column-major (the tensor holds A^T); b = A x* + noise."""
    n, d = c["n"], c["d"]
    g = _generator(seed)
    X = _normal(g, n, d) / math.sqrt(n)
    X *= torch.logspace(0.0, -c["kappa_exp"], d, dtype=torch.float64, device="cuda")
    for _ in range(2):
        X = _hartley_rows(X) * torch.where(
            torch.rand(d, generator=g, device="cuda") < 0.5, -1.0, 1.0).to(torch.float64)
    b = X @ _normal(g, d) + c["noise"] * _normal(g, n)
    return X.t().contiguous(), b


def _batched_shapes(c):
    rng = np.random.default_rng(c["shapes"])
    out = []
    for t in range(c["count"]):
        d = int(rng.integers(c["d_min"], c["d_max"] + 1))
        n = int(max(rng.integers(2000, c["n_max"] + 1), 20 * d))
        out.append(dict(n=n, d=d, per_col=max(8, int(round(rng.uniform(0.005, 0.05) * n))),
                        profile="uniform", scale_exp=4.0, n_dep=0, noise=-1.0))
    return out


class _HostCsc:
    """A host CSC matrix as batched_sparse_spqr reads it (scipy's field names)."""

    def __init__(self, p, i, x, shape):
        self.indptr, self.indices, self.data = p, i, x
        self.shape, self.nnz = shape, x.size

    def tocsc(self):
        return self


def prepare(case, seed):
    c = dict(case)
    s = {"case": c, "seed": 1 + seed % 1000003}
    if c["kind"] == "batched":
        probs = []
        for t, q in enumerate(_batched_shapes(c)):
            p, i, x, b, _ = _sparse_inputs(q, seed * 1009 + 2 * t)
            A = _HostCsc(p.cpu().numpy(), i.cpu().numpy(), x.cpu().numpy(), (q["n"], q["d"]))
            probs.append((A, b.cpu().numpy()))
        s["problems"] = probs
        return s
    if c["kind"] == "dense":
        s["At"], s["b"] = _dense_inputs(c, seed)
    else:
        p, i, x, b, A = _sparse_inputs(c, seed)
        if c["via"] == "host":
            s["A"] = (p.cpu().numpy(), i.cpu().numpy(), x.cpu().numpy(), (c["n"], c["d"]))
            s["b"] = b.cpu().numpy()
            return s
        s["p"], s["i"], s["v"], s["b"] = p, i, x, b
        if c["n_dep"]:
            s["A"] = A
    s["x"] = torch.zeros(c["d"], dtype=torch.float64, device="cuda")
    s["stream"] = torch.cuda.Stream()
    torch.cuda.synchronize()
    return s


# -------------------------------------------------------------------- runs --
def run(s):
    c = s["case"]
    if c["kind"] == "batched":
        xs, infos, _ = skl.batched_sparse_spqr(s["problems"], gamma=c["gamma"], k=c["k"],
                                               it_tol=IT_TOL, seed=s["seed"])
        # one vector of all solutions, and the ranks
        return {"x": np.concatenate(xs), "rank": np.array([q.rank for q in infos])}
    if c["kind"] == "dense":
        args = (c["n"], c["d"], s["At"].data_ptr(), c["n"], s["b"].data_ptr(), s["x"].data_ptr(),
                c["gamma"])
        kw = dict(precision=c["precision"], seed=s["seed"], it_tol=IT_TOL,
                  stream=s["stream"].cuda_stream)
        if c["solver"] == "blendenpik":
            info = skl.dense_blendenpik_device(*args, **kw)
        elif c["solver"] == "nocpqr":
            info = skl.dense_solve_device(*args, c["k"], abs_tol=0.0, rcond=0.0, use_cpqr=0, **kw)
        else:
            info = skl.dense_solve_device(*args, c["k"], **kw)
        return {"x": s["x"], "rank": info.rank}
    if c["via"] == "host":
        r = skl.ls_sparse_spqr(s["A"], s["b"], c["gamma"], c["k"], it_tol=IT_TOL,
                               precision=c["precision"], seed=s["seed"])
        return {"x": r.x, "rank": r.rank}
    info = skl.sparse_solve_device(c["n"], c["d"], s["p"].data_ptr(), s["i"].data_ptr(),
                                   s["v"].data_ptr(), s["b"].data_ptr(), s["x"].data_ptr(),
                                   s["v"].numel(), c["gamma"], c["k"], precision=c["precision"],
                                   seed=s["seed"], it_tol=1e-10 if c["n_dep"] else IT_TOL,
                                   stream=s["stream"].cuda_stream)
    if c["n_dep"]:
        with torch.cuda.stream(s["stream"]):
            return {"fit": s["A"] @ s["x"], "rank": info.rank}
    return {"x": s["x"], "rank": info.rank}


def _work_one(n, d, nnz, gamma, k, dense, it_tol):
    """Input and output bytes, and the operations of the sketch's QR and of the
    LSQR iterations its distortion 1 / sqrt(gamma) asks for."""
    m = math.ceil(gamma * d)
    its = math.log(1 / it_tol) / (0.5 * math.log(gamma))
    in_bytes = 8.0 * nnz if dense else 16.0 * nnz + 8.0 * (d + 1)
    return (in_bytes + 8.0 * (n + d),
            2.0 * d * d * (m - d / 3.0) + 2.0 * k * nnz + its * (4.0 * nnz + 2.0 * d * d))


def work(case):
    c = case
    if c["kind"] == "batched":
        n, d = 0.5 * (2000 + c["n_max"]), 0.5 * (c["d_min"] + c["d_max"])
        b, f = _work_one(n, d, 0.0275 * n * d, c["gamma"], c["k"], False, IT_TOL)
        return {"bytes": c["count"] * b, "flops": c["count"] * f}
    dense = c["kind"] == "dense"
    nnz = float(c["n"]) * c["d"] if dense else float(c["per_col"]) * c["d"]
    b, f = _work_one(c["n"], c["d"], nnz, c["gamma"], c["k"], dense, IT_TOL)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------- exact --
def _refine(A, At, solve, b):
    """Least-squares solution by refinement with solve(g) ~ (A^T A)^-1 g."""
    x = solve(At @ b)
    for _ in range(4):
        x = x + solve(At @ (b - A @ x))
    return x


def _exact_sparse(c, seed):
    p, i, x, b, S = _sparse_inputs(c, seed)
    A = S.to_dense()
    scale = torch.linalg.vector_norm(A, dim=0)
    A /= scale
    L = torch.linalg.cholesky(A.t() @ A)
    y = _refine(A, A.t(), lambda v: torch.cholesky_solve(v[:, None], L)[:, 0], b)
    return y / scale


def _exact_dense(c, seed):
    At, b = _dense_inputs(c, seed)
    A = At.t()
    R = torch.linalg.qr(A, mode="r").R

    def solve(v):
        w = torch.linalg.solve_triangular(R.t(), v[:, None], upper=False)
        return torch.linalg.solve_triangular(R, w, upper=True)[:, 0]

    return _refine(A, At, solve, b)


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "batched":
        xs = [_exact_sparse(q, seed * 1009 + 2 * t) for t, q in enumerate(_batched_shapes(c))]
        return {"x": torch.cat(xs).cpu().numpy(), "rank": None}
    if c.get("n_dep") or float(c["n"]) * c["d"] * c["d"] > 3.1e12:
        return None          # x is not unique, or would take minutes
    x = _exact_dense(c, seed) if c["kind"] == "dense" else _exact_sparse(c, seed)
    return {"x": x.cpu().numpy() if c.get("via") == "host" else x, "rank": None}
