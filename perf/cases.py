"""Performance cases of the framework, each one call (or one short sequence of calls) a program makes through the
public Python API: KernelMatrix products in every storage type and for one to 256 right-hand sides, batched
products, gradients, the construction of a KernelMatrix, products with a user-assembled HierarchicalMatrix and the
hierarchical Cholesky with its solve.

``listed()`` gives the fixed cases and ``draw(rng)`` further ones of the same ranges; ``prepare`` makes what a
program has in hand before the call, ``run`` makes the call, ``work`` counts what it cannot do without and
``exact`` gives the result in plain FP64.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "hierarchicalmatrices.jl_gb300"))

import hierarchicalmatrices as hm  # noqa: E402

DEV = "cuda"
KERNEL = {"cauchy": "cauchykernel", "coulomb": "coulombkernel", "coulombprime": "coulombprimekernel",
          "log": "logkernel"}
VECTOR = {"f64": torch.float64, "f32": torch.float32, "df64": torch.float64}
STORAGE = {"f64": np.float64, "f32": np.float32, "df64": "df64"}
RANK = 20


def _product(name, kernel, points, n, m, dtype, k, transposed=False):
    return {"name": name, "kind": "product", "kernel": kernel, "points": points, "n": n, "m": m, "dtype": dtype,
            "k": k, "transposed": transposed}


def listed():
    return [
        # the size of the reference's worked example (Chebyshev points, FP64): latency and launches
        _product("example_f64", "cauchy", "chebyshev", 1000, 1000, "f64", 1),
        # the FP32 product of a large grid, one right-hand side: the benchmark's workload
        _product("grid_f32", "cauchy", "grid", 1 << 20, 1 << 20, "f32", 1),
        # the same in FP64, the reference's own precision
        _product("grid_f64", "cauchy", "grid", 1 << 20, 1 << 20, "f64", 1),
        # clustered points (a deep, uneven tree) with double-float storage, an odd size
        _product("beta_df64", "cauchy", "beta", 300007, 300007, "df64", 1),
        # an ordinary rectangular matrix of odd sizes between two random point sets, a few vectors
        _product("rect_log_f32_k3", "log", "uniform", 100003, 77777, "f32", 3),
        # a block of vectors, as in a block Krylov method
        _product("block32_f32", "cauchy", "grid", 1 << 19, 1 << 19, "f32", 32),
        # many vectors at once: a KernelMatrix applied to a dense matrix
        _product("block256_f32", "cauchy", "grid", 1 << 18, 1 << 18, "f32", 256),
        # many independent matrices of uneven sizes in one product
        {"name": "batch_f32_k8", "kind": "batch", "instances": 128, "lo": 1024, "hi": 65536, "dtype": "f32", "k": 8},
        # a training step's loss and gradients in the weights and both point sets
        {"name": "grad_f32", "kind": "grad", "n": 65536, "dtype": "f32"},
        # compression of a new point set and its first product
        {"name": "build_f64", "kind": "build", "kernel": "cauchy", "points": "uniform", "n": 131072, "m": 131072,
         "dtype": "f64"},
        # a user-assembled HierarchicalMatrix (low-rank and dense blocks) times a vector
        {"name": "hodlr_f64", "kind": "hodlr", "n": 16384, "leaf": 64, "dtype": "f64", "k": 1},
        # factorisation of a symmetric positive definite HierarchicalMatrix and the solve with its factor
        {"name": "cholesky_f64", "kind": "cholesky", "n": 8192, "leaf": 64, "k": 4},
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product"] * 6 + ["batch", "grad", "build", "hodlr", "cholesky"])
    if kind == "product":
        dtype = rng.choice(["f64", "f32", "f32", "df64"])
        points = rng.choice(["grid", "grid", "uniform", "beta", "chebyshev", "quadratic"])
        kernel = rng.choice(["cauchy", "cauchy", "log", "coulomb", "coulombprime"])
        if points in ("uniform", "beta") and kernel == "coulombprime":
            kernel = "cauchy"            # the closest pairs of random points overflow FP32 panels
        k = rng.choice([1, 1, 1, 2, 3, 5, 8, 13, 16, 32, 48, 64, 100, 128, 256])
        most = {"grid": 1 << 20, "uniform": 300007, "beta": 300007, "chebyshev": 1 << 17, "quadratic": 1 << 17}[points]
        n = _log_size(rng, 500, min(most, (1 << (26 if dtype == "f32" else 22)) // k))
        m = n if points != "uniform" else max(500, min(n, int(n * rng.uniform(0.3, 1.0))))
        transposed = rng.random() < 0.2
        case = _product("", kernel, points, n, m, dtype, k, transposed)
        del case["name"]
        return case
    if kind == "batch":
        return {"kind": "batch", "instances": rng.randint(16, 120), "lo": 1024, "hi": _log_size(rng, 4096, 65536),
                "dtype": rng.choice(["f32", "f32", "f64"]), "k": rng.choice([1, 2, 4, 8])}
    if kind == "grad":
        return {"kind": "grad", "n": _log_size(rng, 1000, 120000), "dtype": rng.choice(["f32", "f64"])}
    if kind == "build":
        n = _log_size(rng, 1000, 131072)
        return {"kind": "build", "kernel": rng.choice(["cauchy", "log"]), "points": "uniform", "n": n,
                "m": max(500, int(n * rng.uniform(0.5, 1.0))), "dtype": rng.choice(["f64", "f32", "df64"])}
    if kind == "hodlr":
        return {"kind": "hodlr", "n": _log_size(rng, 512, 16384), "leaf": rng.choice([32, 64, 100]),
                "dtype": rng.choice(["f64", "f32"]), "k": rng.choice([1, 1, 4, 16])}
    return {"kind": "cholesky", "n": _log_size(rng, 512, 8192), "leaf": rng.choice([32, 64, 80]),
            "k": rng.randint(1, 8)}


# ---------------------------------------------------------------- points (non-increasing, with their box)

def _chebyshev(n, kind):
    i = np.arange(n, dtype=np.float64)
    p = np.cos((2 * i + 1) * (np.pi / (2 * n))) if kind == 1 else np.cos(i * (np.pi / (n - 1)))
    return np.clip(p, -1.0, 1.0)


def _spread(p, gap=1e-9):
    """Sorted values raised so that neighbours are at least `gap` apart, descending."""
    steps = np.arange(p.size, dtype=np.float64) * gap
    return (np.maximum.accumulate(np.sort(p) - steps) + steps)[::-1].copy()


def _points(family, n, m, rng):
    """(x, y, a, b, c, d): n row points in [b, a], m column points in [d, c]."""
    if family == "grid":                        # interleaved: x halfway between the y
        return ((np.arange(n) / n + 1 / (2 * n))[::-1].copy(), (np.arange(m) / m)[::-1].copy(), 1.0, 0.0, 1.0, 0.0)
    if family == "uniform":
        return np.sort(rng.random(n))[::-1].copy(), np.sort(rng.random(m))[::-1].copy(), 1.0, 0.0, 1.0, 0.0
    if family == "beta":                        # Beta(1/2, 1/2): clustered at both ends
        x, y = _spread(rng.beta(0.5, 0.5, n)), _spread(rng.beta(0.5, 0.5, m))
        top = max(1.0, x[0], y[0])
        return x, y, top, 0.0, top, 0.0
    if family == "chebyshev":                   # x first kind, y second kind
        return _chebyshev(n, 1), _chebyshev(m, 2), 1.0, -1.0, 1.0, -1.0
    if family == "quadratic":                   # x_i = i(i+1), y_i = (i+1/2)(i+3/2), scaled to [0, 1]
        i, j = np.arange(n, 0, -1, dtype=np.float64), np.arange(m, 0, -1, dtype=np.float64)
        top = (m + 0.5) * (m + 1.5)
        return i * (i + 1) / top, (j + 0.5) * (j + 1.5) / top, 1.0, 0.0, 1.0, 0.0
    raise ValueError(family)


def _case_points(case, seed):
    return _points(case["points"], case["n"], case["m"], np.random.default_rng(seed))


def _batch_points(case, seed):
    """Point sets of the instances: the sizes belong to the case, log-uniform in [lo, hi]; the points to the seed."""
    sizes = np.random.default_rng([case["instances"], case["lo"], case["hi"]])
    ns = np.exp(sizes.uniform(np.log(case["lo"]), np.log(case["hi"]), case["instances"])).astype(np.int64)
    rng = np.random.default_rng(seed)
    return ([np.sort(rng.random(n))[::-1].copy() for n in ns], [np.sort(rng.random(n))[::-1].copy() for n in ns])


def _vectors(rows, k, dtype, seed):
    """N(0, 1) right-hand sides: a vector, or k columns stored column-major."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    v = torch.randn((k, rows), generator=g, device=DEV, dtype=dtype)
    return v[0] if k == 1 else v.t()


# ---------------------------------------------------------------- a smooth-kernel HODLR matrix

LENGTH, SHIFT, TOL, NODES = 0.15, 1e-2, 1e-12, 32


def _gauss(x, y):
    d = x[:, None] - y[None, :]
    return np.exp(-d * d / (2 * LENGTH * LENGTH))


def _interpolation(p):
    """(Chebyshev nodes of [min p, max p], Lagrange basis at p)."""
    lo, hi = p.min(), p.max()
    theta = (2 * np.arange(NODES) + 1) * (np.pi / (2 * NODES))
    t = np.clip((2 * p - lo - hi) / max(hi - lo, 1e-300), -1.0, 1.0)
    basis = np.cos(np.arccos(t)[:, None] * np.arange(NODES)) @ (np.cos(np.arange(NODES)[:, None] * theta) * (2 / NODES)
                                                             * np.where(np.arange(NODES) == 0, 0.5, 1.0)[:, None])
    return (lo + hi) / 2 + (hi - lo) / 2 * np.cos(theta), basis


def _hodlr_blocks(n, leaf, seed):
    """K + SHIFT I for the Gaussian kernel on n sorted uniform points, halved down to `leaf` rows: a nested
    (left, (U, sigma, V), right) tree with dense diagonal leaves, on the host."""
    x = np.sort(np.random.default_rng(seed).random(n))

    def half(p, q):
        if p.size <= NODES or q.size <= NODES:
            u, s, vt = np.linalg.svd(_gauss(p, q), full_matrices=False)
        else:
            (tp, bp), (tq, bq) = _interpolation(p), _interpolation(q)
            (qp, rp), (qq, rq) = np.linalg.qr(bp), np.linalg.qr(bq)
            u, s, vt = np.linalg.svd(rp @ _gauss(tp, tq) @ rq.T)
            u, vt = qp @ u, (qq @ vt.T).T
        r = int((s > TOL * s[0]).sum())
        return u[:, :r], s[:r], vt[:r].T

    def build(i, j):
        if j - i <= leaf:
            return _gauss(x[i:j], x[i:j]) + SHIFT * np.eye(j - i)
        mid = (i + j) // 2
        return build(i, mid), half(x[i:mid], x[mid:j]), build(mid, j)

    return build(0, n)


def _column_major(a, dtype):
    return torch.tensor(np.ascontiguousarray(a.T), dtype=dtype, device=DEV).t()


def _tree(blocks, dtype, lower):
    if isinstance(blocks, np.ndarray):
        return _column_major(blocks, dtype)
    left, (u, s, v), right = blocks
    U, S, V = _column_major(u, dtype), torch.tensor(s, dtype=dtype, device=DEV), _column_major(v, dtype)
    H = hm.HierarchicalMatrix(2, 2)
    H[hm.Block(1), hm.Block(1)] = _tree(left, dtype, lower)
    H[hm.Block(1), hm.Block(2)] = hm.LowRankMatrix(U, S, V)
    if lower:
        H[hm.Block(2), hm.Block(1)] = hm.LowRankMatrix(V, S, U)
    H[hm.Block(2), hm.Block(2)] = _tree(right, dtype, lower)
    return H


def _dense(blocks, dtype):
    """The symmetric dense matrix of the blocks, rounded to `dtype` as the tree stores them, in FP64."""
    def rounded(a):
        return torch.tensor(np.ascontiguousarray(a), device=DEV).to(dtype).double()

    def size(b):
        return b.shape[0] if isinstance(b, np.ndarray) else size(b[0]) + size(b[2])

    D = torch.zeros((size(blocks),) * 2, dtype=torch.float64, device=DEV)

    def fill(b, at):
        if isinstance(b, np.ndarray):
            D[at:at + b.shape[0], at:at + b.shape[0]] = rounded(b)
            return b.shape[0]
        left, (u, s, v), right = b
        n1 = fill(left, at)
        n2 = fill(right, at + n1)
        M = (rounded(u) * rounded(s)) @ rounded(v).t()
        D[at:at + n1, at + n1:at + n1 + n2] = M
        D[at + n1:at + n1 + n2, at:at + n1] = M.t()
        return n1 + n2

    fill(blocks, 0)
    return D


# ---------------------------------------------------------------- prepare and run

def _kernel_matrix(case, points):
    return hm.KernelMatrix(getattr(hm, KERNEL[case["kernel"]]), *points, dtype=STORAGE[case["dtype"]])


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "product":
        state["H"] = _kernel_matrix(case, _case_points(case, seed))
        rows = case["n"] if case["transposed"] else case["m"]
        state["v"] = _vectors(rows, case["k"], VECTOR[case["dtype"]], seed)
    elif kind == "batch":
        xs, ys = _batch_points(case, seed)
        state["H"] = hm.KernelMatrixBatch(hm.cauchykernel, xs, ys, [(1.0, 0.0, 1.0, 0.0)] * len(xs),
                                          dtype=STORAGE[case["dtype"]])
        state["v"] = _vectors(state["H"].shape[1], case["k"], VECTOR[case["dtype"]], seed)
    elif kind == "grad":
        x, y, *box = _points("uniform", case["n"], case["n"], np.random.default_rng(seed))
        state["H"] = hm.KernelMatrix(hm.cauchykernel, x, y, *box, dtype=STORAGE[case["dtype"]])
        state["w"], state["t"] = (_vectors(case["n"], 1, VECTOR[case["dtype"]], seed + s) for s in (0, 7))
    elif kind == "build":
        state["points"] = _case_points(case, seed)
        state["v"] = _vectors(case["m"], 1, VECTOR[case["dtype"]], seed)
    elif kind == "hodlr":
        state["H"] = _tree(_hodlr_blocks(case["n"], case["leaf"], seed), VECTOR[case["dtype"]], lower=True)
        state["v"] = _vectors(case["n"], case["k"], VECTOR[case["dtype"]], seed)
    elif kind == "cholesky":
        state["H"] = _tree(_hodlr_blocks(case["n"], case["leaf"], seed), torch.float64, lower=False)
        state["v"] = _vectors(case["n"], case["k"], torch.float64, seed)
    else:
        raise ValueError(kind)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "product" and case["transposed"]:
        return state["H"].T @ state["v"]
    if kind in ("product", "batch", "hodlr"):
        return state["H"] @ state["v"]
    if kind == "grad":
        return state["H"].loss_and_grad(state["w"], state["t"])
    if kind == "build":
        return _kernel_matrix(case, state["points"]) @ state["v"]
    R = hm.hierarchicalcholesky(state["H"])
    return hm.solvetransposed(R, state["v"])


# ---------------------------------------------------------------- work

def _element(dtype):
    return 4 if dtype == "f32" else 8


def _stored(points):
    """Values of the compressed matrix: near-field entries, leaf bases and far-field cores."""
    return hm.Plan(*points).sizes["stored_values"]


def _hodlr_values(n, leaf, rank=12):
    """(off-diagonal factor values of one triangle, dense leaf values) at the blocks' usual rank."""
    if n <= leaf:
        return 0, n * n
    (l1, d1), (l2, d2) = _hodlr_values(n // 2, leaf, rank), _hodlr_values(n - n // 2, leaf, rank)
    return l1 + l2 + rank * n, d1 + d2


def work(case):
    kind, k, es = case["kind"], case.get("k", 1), _element(case.get("dtype", "f64"))
    if kind in ("product", "build"):
        stored = _stored(_case_points(case, 0))
        vectors = (case["n"] + case["m"]) * k
        if kind == "build":                    # every value evaluated and written once, then read by the product
            return {"bytes": 2 * stored * es + vectors * es, "flops": 8 * stored}
        return {"bytes": (stored + vectors) * es, "flops": 2 * stored * k}
    if kind == "batch":
        xs, ys = _batch_points(case, 0)
        stored = sum(_stored((x, y, 1.0, 0.0, 1.0, 0.0)) for x, y in zip(xs, ys))
        return {"bytes": (stored + 2 * sum(map(len, xs)) * k) * es, "flops": 2 * stored * k}
    if kind == "grad":
        stored = _stored(_points("uniform", case["n"], case["n"], np.random.default_rng(0)))
        return {"bytes": (4 * stored + 9 * case["n"]) * es, "flops": 8 * stored}
    low, dense = _hodlr_values(case["n"], case["leaf"])
    if kind == "hodlr":
        return {"bytes": (2 * low + dense + 2 * case["n"] * k) * es, "flops": 2 * (2 * low + dense) * k}
    # factorisation: per tree level a solve, a Gram matrix and an update of every block below, rank 12
    n, leaf, r = case["n"], case["leaf"], 12
    levels = max(1, math.ceil(math.log2(n / leaf)))
    return {"bytes": 8 * (2 * (low + dense) + 2 * n * k),
            "flops": n * leaf * leaf / 3 + levels * levels * n * 20 * r * r + 2 * (low + dense) * k}


# ---------------------------------------------------------------- exact results

def _f(kernel, d):
    if kernel == "cauchy":
        return 1.0 / d
    if kernel == "coulomb":
        return 1.0 / (d * d)
    if kernel == "coulombprime":
        return 1.0 / (d * d * d)
    return torch.log(torch.abs(d))


def _df(kernel, d):
    """The kernel's derivative in x - y."""
    if kernel != "cauchy":
        raise ValueError(kernel)
    return -1.0 / (d * d)


def _dense_apply(f, x, y, v, kernel="cauchy"):
    """sum_j f(x_i - y_j) v_j in FP64, a slice of rows at a time."""
    x, y = (torch.tensor(np.ascontiguousarray(p), device=DEV) for p in (x, y))
    v = v.double()
    out = torch.empty((x.numel(),) + tuple(v.shape[1:]), dtype=torch.float64, device=DEV)
    step = max(1, (1 << 27) // y.numel())
    for i in range(0, x.numel(), step):
        out[i:i + step] = f(kernel, x[i:i + step, None] - y[None, :]) @ v
    return out


def _grid_apply(kernel, n, v, transposed):
    """The same on the interleaved grid of a power of two (whose points are exact in FP64), where x_i - y_j =
    (j - i + 1/2) / n is a Toeplitz matrix, by FFT."""
    d = (torch.arange(2 * n, device=DEV, dtype=torch.float64) - n + 0.5) / n      # x_i - y_j at j - i + n
    t = _f(kernel, d)
    t[0] = 0.0
    if not transposed:
        t = t.flip(0).roll(1)              # at i - j + n
    t = torch.fft.rfft(t.roll(n))
    v = v.double().reshape(n, -1)
    out = [torch.fft.irfft(t * torch.fft.rfft(v[:, q].contiguous(), n=2 * n), n=2 * n)[:n] for q in range(v.shape[1])]
    return torch.stack(out, 1)


def _exact_product(case, seed):
    rows = case["n"] if case["transposed"] else case["m"]
    v = _vectors(rows, case["k"], VECTOR[case["dtype"]], seed)
    if case["points"] == "grid" and case["n"] & (case["n"] - 1) == 0:
        u = _grid_apply(case["kernel"], case["n"], v, case["transposed"])
        return u[:, 0] if case["k"] == 1 else u
    pairs = case["n"] * case["m"]
    if pairs > 1.5e11 or pairs * case["k"] > 2e12:
        return None
    x, y, *_ = _case_points(case, seed)
    if case["transposed"]:                     # f(x - y) read by columns: f(-(y - x))
        return _dense_apply(lambda kernel, d: _f(kernel, -d), y, x, v, case["kernel"])
    return _dense_apply(_f, x, y, v, case["kernel"])


def exact(case, seed):
    kind = case["kind"]
    if kind == "product":
        return _exact_product(case, seed)
    if kind == "batch":
        xs, ys = _batch_points(case, seed)
        v = _vectors(sum(map(len, ys)), case["k"], VECTOR[case["dtype"]], seed)
        out, at = [], 0
        for x, y in zip(xs, ys):
            out.append(_dense_apply(_f, x, y, v[at:at + len(y)]))
            at += len(y)
        return torch.cat(out)
    if kind == "grad":
        x, y, *_ = _points("uniform", case["n"], case["n"], np.random.default_rng(seed))
        w, t = (_vectors(case["n"], 1, VECTOR[case["dtype"]], seed + s).double() for s in (0, 7))
        r = _dense_apply(_f, x, y, w) - t
        gw = -_dense_apply(_f, y, x, r)
        gx = r * _dense_apply(_df, x, y, w)
        gy = -w * _dense_apply(_df, y, x, r)
        return float(0.5 * torch.dot(r, r)), gw, gx, gy
    if kind == "build":
        if case["n"] * case["m"] > 1.5e11:
            return None
        x, y, *_ = _case_points(case, seed)
        return _dense_apply(_f, x, y, _vectors(case["m"], 1, VECTOR[case["dtype"]], seed), case["kernel"])
    D = _dense(_hodlr_blocks(case["n"], case["leaf"], seed), VECTOR[case.get("dtype", "f64")])
    v = _vectors(case["n"], case["k"], VECTOR[case.get("dtype", "f64")], seed).double()
    if kind == "hodlr":
        return D @ v
    L = torch.linalg.cholesky(D)
    u = torch.linalg.solve_triangular(L, v.reshape(case["n"], -1), upper=False)
    return u if case["k"] > 1 else u[:, 0]
