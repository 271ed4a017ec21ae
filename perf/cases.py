"""What a user of this library has it do, as cases that can be timed.

A case is a dict of plain values.  Kinds:

lu      a new matrix and right-hand sides through one LinearCache: cache.A = A,
        then one solve! per right-hand side (one getrf, `nrhs` getrs).
solve   a new right-hand side block against a cache whose factors are resident
        (`nrhs` columns in one solve!; adjoint: A^T x = b).
mixed   a new matrix and right-hand sides with low-precision factors and FP64
        refinement (GB300MixedLUFactorization).
batch   uneven systems packed back to back, solved by one Batch.solve.
serve   a burst of requests to the serving loop, each a new matrix of its key
        (30 %) or a right-hand side for the key's current matrix.

Sizes and matrices are those of the benchmark configurations (iid N(0,1),
G + 4 sqrt(n) I, singular values 1..1e6, I - g J with n in 8..256, and a stream
of sizes log-uniform up to 4096).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()


def listed():
    return [
        # a small system of an integrator's Newton step: latency and launches
        {"name": "lu_n96_host", "kind": "lu", "n": 96, "nrhs": 1, "solve": "exact", "where": "host"},
        # the plain FP64 configuration: n = 1000, one right-hand side, host arrays
        {"name": "lu_n1000_host", "kind": "lu", "n": 1000, "nrhs": 1, "solve": "exact", "where": "host"},
        # the cached FP64 configuration: one getrf and 16 successive getrs
        {"name": "lu_n8192_16rhs", "kind": "lu", "n": 8192, "nrhs": 16, "solve": "exact", "where": "device"},
        # a new b on resident factors, host vector
        {"name": "solve_n2000_host", "kind": "solve", "n": 2000, "nrhs": 1, "solve": "exact",
         "adjoint": False, "where": "host"},
        # an adjoint pass with several right-hand sides at a ragged order, fast sweeps
        {"name": "solve_n6001_adjoint_5rhs", "kind": "solve", "n": 6001, "nrhs": 5, "solve": "fast",
         "adjoint": True, "where": "device"},
        # the default algorithm for well-conditioned matrices (FP32 LU + IR)
        {"name": "mixed_fp32_n3001", "kind": "mixed", "n": 3001, "nrhs": 1, "factor": "fp32",
         "pivot": "partial", "refine": "ir", "matrix": "shifted"},
        # the mixed-precision configuration: tensor-core updates, n = 16384, 4 RHS
        {"name": "mixed_bf16_n16384_4rhs", "kind": "mixed", "n": 16384, "nrhs": 4, "factor": "bf16",
         "pivot": "partial", "refine": "ir", "matrix": "shifted"},
        # no pivoting after the butterfly transform, FP16 operands, ragged order
        {"name": "mixed_fp16_rbt_n6002_2rhs", "kind": "mixed", "n": 6002, "nrhs": 2, "factor": "fp16",
         "pivot": "rbt", "refine": "ir", "matrix": "shifted"},
        # the hard configuration: condition number 1e6, FP32 LU + GMRES-IR
        {"name": "mixed_gmres_n3000_4rhs", "kind": "mixed", "n": 3000, "nrhs": 4, "factor": "fp32",
         "pivot": "partial", "refine": "gmres_ir", "matrix": "svd"},
        # the batched configuration, FP64 and FP32 + IR
        {"name": "batch_fp64_20000", "kind": "batch", "count": 20000, "nmax": 256, "precision": "fp64"},
        {"name": "batch_fp32_20000", "kind": "batch", "count": 20000, "nmax": 256, "precision": "fp32"},
        # the served stream's mix, everything submitted at once
        {"name": "serve_48", "kind": "serve", "requests": 48, "keys": 24, "nmax": 2048},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lu", "lu", "solve", "mixed", "mixed", "batch", "serve"])
    if kind == "lu":
        n = _log_int(rng, 64, 7000)
        where = "host" if n <= 2000 else "device"
        return {"kind": kind, "n": n, "nrhs": rng.choice([1, 1, 2, 4, 16]), "solve": rng.choice(["exact", "exact", "fast"]),
                "where": where}
    if kind == "solve":
        n = _log_int(rng, 64, 7000)
        where = "host" if n <= 2000 else "device"
        return {"kind": kind, "n": n, "nrhs": rng.randint(1, 12), "solve": rng.choice(["exact", "fast"]),
                "adjoint": rng.random() < 0.4, "where": where}
    if kind == "mixed":
        if rng.random() < 0.2:
            return {"kind": kind, "n": _log_int(rng, 500, 4000), "nrhs": rng.randint(1, 4), "factor": "fp32",
                    "pivot": "partial", "refine": "gmres_ir", "matrix": "svd"}
        factor = rng.choice(["fp32", "bf16", "fp16"])
        return {"kind": kind, "n": _log_int(rng, 300, 8000 if factor == "fp32" else 16000), "nrhs": rng.randint(1, 6),
                "factor": factor, "pivot": rng.choice(["partial", "partial", "rbt"]), "refine": "ir",
                "matrix": "shifted"}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 100, 18000), "nmax": _log_int(rng, 32, 256),
                "precision": rng.choice(["fp64", "fp32"])}
    requests = rng.randint(16, 64)
    return {"kind": kind, "requests": requests, "keys": max(8, requests // 2), "nmax": _log_int(rng, 500, 2500)}


# ---------------------------------------------------------------------------
# inputs

class TorchMatrix(pkg.DeviceMatrix):
    """A column-major view of a torch CUDA tensor that holds the transpose:
    row j of the tensor is column j of the matrix."""

    def __init__(self, t: torch.Tensor):
        assert t.is_cuda and t.is_contiguous() and t.dim() == 2
        self.cols, self.rows = t.shape
        self.dtype = np.dtype(np.float64)
        self.ld = self.rows
        self.nbytes = t.numel() * 8
        self.ptr = t.data_ptr()
        self._owner = False
        self._tensor = t


def _randn(gen, *shape):
    return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=gen)


def _matrix(gen, n, which):
    """The transpose of the case's matrix (so its memory is column-major)."""
    if which == "svd":
        s = torch.logspace(0.0, 6.0, n, dtype=torch.float64, device="cuda")
        q1, _ = torch.linalg.qr(_randn(gen, n, n))
        q2, _ = torch.linalg.qr(_randn(gen, n, n))
        return ((q2 * s) @ q1.T).contiguous()
    at = _randn(gen, n, n)
    if which == "shifted":
        at.diagonal().add_(4.0 * math.sqrt(n))
    return at


def _dense_inputs(case, seed):
    """(A^T, B^T): torch tensors on the GPU, row j = column j."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"]
    return _matrix(gen, n, case.get("matrix", "plain")), _randn(gen, case["nrhs"], n)


def _batch_inputs(case, seed):
    # the sizes belong to the case (a batch object is made for them), the values to the seed
    sizes = np.random.default_rng(case["count"]).integers(8, case["nmax"] + 1, size=case["count"]).astype(np.int64)
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = torch.from_numpy(sizes).cuda()
    gamma = torch.from_numpy(rng.uniform(0.01, 0.5, size=case["count"])).cuda()
    A = _randn(gen, int((sizes ** 2).sum()))
    A *= torch.repeat_interleave(-gamma / n.double().sqrt(), n * n)
    # the diagonals: system i's entry j lies at a_off[i] + j (n_i + 1)
    a_off = torch.cumsum(n * n, 0) - n * n
    x_off = torch.cumsum(n, 0) - n
    j = torch.arange(int(sizes.sum()), device="cuda") - torch.repeat_interleave(x_off, n)
    A[torch.repeat_interleave(a_off, n) + j * torch.repeat_interleave(n + 1, n)] += 1.0
    return sizes, A, _randn(gen, int(sizes.sum()))


def _serve_inputs(case, seed):
    """Per key: n and its first matrix; then the requests (key, b, A or None)."""
    shape = np.random.default_rng(case["requests"])  # sizes and order of the burst belong to the case
    sizes = np.round(np.exp(shape.uniform(math.log(64), math.log(case["nmax"]), size=case["keys"]))).astype(int)
    rng = np.random.default_rng(seed)

    def shifted(n):
        a = np.asfortranarray(rng.standard_normal((n, n)))
        a[np.diag_indices(n)] += 4.0 * math.sqrt(n)
        return a

    first = [shifted(int(n)) for n in sizes]
    # 60 % of the keys get a new matrix, with their first request of the burst
    # (so every pass over the burst solves the same systems); at two requests
    # per key 30 % of the requests factor
    renewed = shape.random(case["keys"]) < 0.6
    requests, seen = [], set()
    for _ in range(case["requests"]):
        k = int(shape.integers(case["keys"]))
        n = int(sizes[k])
        requests.append((k, rng.standard_normal(n), shifted(n) if renewed[k] and k not in seen else None))
        seen.add(k)
    return first, requests


# ---------------------------------------------------------------------------
# states

class Dense:
    def __init__(self, case, seed):
        at, bt = _dense_inputs(case, seed)
        self.kind, self.adjoint = case["kind"], case.get("adjoint", False)
        if case["kind"] == "mixed":
            alg = pkg.GB300MixedLUFactorization(factor=case["factor"], refine=case["refine"], pivot=case["pivot"])
        else:
            alg = pkg.GB300LUFactorization(solve=case["solve"])
        self.host = case.get("where") == "host"
        nrhs = case["nrhs"]
        # "lu" solves its right-hand sides one after another, the others in one block
        split = [slice(j, j + 1) for j in range(nrhs)] if self.kind == "lu" else [slice(0, nrhs)]
        if self.host:
            self.A = np.asfortranarray(at.cpu().numpy().T)
            self.bs = [np.asfortranarray(bt[s].cpu().numpy().T) for s in split]
            if nrhs == 1 or self.kind == "lu":
                self.bs = [np.ascontiguousarray(b[:, 0]) for b in self.bs]
            self.us = [np.zeros_like(b) for b in self.bs]
        else:
            self.A = TorchMatrix(at)
            self.xt = torch.empty_like(bt)
            self.bs = [TorchMatrix(bt[s]) for s in split]
            self.us = [TorchMatrix(self.xt[s]) for s in split]
        torch.cuda.synchronize()
        alias = pkg.LinearAliasSpecifier(alias_A=True, alias_b=True)
        self.cache = pkg.init(pkg.LinearProblem(self.A, self.bs[0]), alg, alias=alias)
        if self.kind == "solve":
            self.cache.u = self.us[0]
            pkg.solve_bang(self.cache)

    def run(self):
        cache = self.cache
        if self.kind != "solve":
            cache.A = self.A
        for b, u in zip(self.bs, self.us):
            cache.b = b
            cache.u = u
            sol = pkg.solve_bang(cache, adjoint=self.adjoint)
            if not pkg.successful_retcode(sol):
                raise RuntimeError("the solve failed: %s" % sol.retcode)
        return list(self.us) if self.host else self.xt

    def __del__(self):
        try:
            self.cache.cacheval.close()
        except Exception:
            pass


class Batched:
    def __init__(self, case, seed):
        sizes, self.A, self.b = _batch_inputs(case, seed)
        self.x = torch.empty_like(self.b)
        torch.cuda.synchronize()
        self.batch = pkg.Batch(pkg.default_context(), sizes, case["precision"])

    def run(self):
        self.x.copy_(self.b)
        torch.cuda.current_stream().synchronize()  # the library works on a stream of its own
        self.batch.solve(TorchMatrix(self.A.view(1, -1)), TorchMatrix(self.x.view(1, -1)))
        return [self.x, self.batch.info]

    def __del__(self):
        try:
            self.batch.close()
        except Exception:
            pass


class Served:
    def __init__(self, case, seed):
        from linearsolve_gb300.serving import Server
        first, self.requests = _serve_inputs(case, seed)
        self.server = Server(pkg.default_context(), workers=4, precision="fp32", solve="fast")
        for k, a in enumerate(first):
            self.server.submit(k, k, np.ones(a.shape[0]), a)
        self._collect(len(first))

    def _collect(self, count):
        got = {}
        while len(got) < count:
            for d in self.server.poll(256, wait_ms=20):
                if d["status"] != 0:
                    raise RuntimeError("request %d failed with status %d" % (d["tag"], d["status"]))
                got[d["tag"]] = d["x"]
        return [got[i] for i in range(count)]

    def run(self):
        for i, (k, b, a) in enumerate(self.requests):
            self.server.submit(i, k, b, a)
        return np.concatenate(self._collect(len(self.requests)))

    def __del__(self):
        try:
            self.server.close()
        except Exception:
            pass


def prepare(case, seed):
    if case["kind"] == "batch":
        return Batched(case, seed)
    if case["kind"] == "serve":
        return Served(case, seed)
    return Dense(case, seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------------------
# work and 64-bit results

def _lu_flops(n):
    return 2.0 * n ** 3 / 3.0


def _mean_power(nmin, nmax, p):
    k = np.arange(nmin, nmax + 1, dtype=np.float64)
    return float((k ** p).mean())


def work(case):
    if case["kind"] == "batch":
        c = case["count"]
        m1, m2, m3 = (_mean_power(8, case["nmax"], p) for p in (1, 2, 3))
        return {"bytes": c * (8.0 * m2 + 16.0 * m1), "flops": c * (2.0 * m3 / 3.0 + 2.0 * m2)}
    if case["kind"] == "serve":
        # sizes log-uniform in [64, nmax]: E[n^p] = (nmax^p - 64^p) / (p ln(nmax / 64))
        r, ln = case["requests"], math.log(case["nmax"] / 64.0)
        m2, m3 = ((case["nmax"] ** p - 64.0 ** p) / (p * ln) for p in (2, 3))
        return {"bytes": 8.0 * r * m2, "flops": r * (0.3 * 2.0 * m3 / 3.0 + 2.0 * m2)}
    n, w = float(case["n"]), case["nrhs"]
    flops = 2.0 * n * n * w + (0.0 if case["kind"] == "solve" else _lu_flops(n))
    return {"bytes": 8.0 * n * n + 16.0 * n * w, "flops": flops}


def exact(case, seed):
    if case["kind"] == "batch":
        sizes, A, b = _batch_inputs(case, seed)
        n = torch.from_numpy(sizes).cuda()
        a_off, x_off = torch.cumsum(n * n, 0) - n * n, torch.cumsum(n, 0) - n
        x = torch.empty_like(b)
        for k in np.unique(sizes):
            k = int(k)
            which = (n == k).nonzero()[:, 0]
            at = A[a_off[which][:, None] + torch.arange(k * k, device="cuda")].view(-1, k, k)
            at_idx = x_off[which][:, None] + torch.arange(k, device="cuda")
            x[at_idx] = torch.linalg.solve(at.transpose(1, 2), b[at_idx])
        return [x, None]
    if case["kind"] == "serve":
        current, requests = _serve_inputs(case, seed)
        xs = []
        for k, b, a in requests:
            if a is not None:
                current[k] = a
            xs.append(torch.linalg.solve(torch.from_numpy(current[k]).cuda(), torch.from_numpy(b).cuda()).cpu().numpy())
        return np.concatenate(xs)
    at, bt = _dense_inputs(case, seed)
    x = torch.linalg.solve(at if case.get("adjoint") else at.T, bt.T).T
    if case.get("where") != "host":
        return x.contiguous()
    x = x.cpu().numpy()
    if case["kind"] == "lu":
        return [np.ascontiguousarray(x[j]) for j in range(case["nrhs"])]
    return [np.ascontiguousarray(x[0] if case["nrhs"] == 1 else x.T)]
