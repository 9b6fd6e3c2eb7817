"""The work that users of this solver have it do, as timed cases.

Each case is one call (or one solve) through the public Python binding
(`sipg_gb300`): the operator apply in FP64 and FP32, the host-buffer apply, the
right-hand side, plain FP64 CG, the mixed-precision solve, a batch of uneven
problems, and a burst of requests to the solve server.  Sizes are those of the
benchmark configurations and the tests (16 x 16 up to 1024 x 1024 elements,
degrees 1..8), with odd ones among them.
"""
import importlib
import math
import os
import sys

import numpy as np
import torch

PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-sipg-matrix-free_gb300")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)
sipg = importlib.import_module("sipg_gb300")

# Solves compared with a direct 64-bit solve up to this many nodes per axis.
EXACT_SOLVE_NODES = 3600


def listed():
    return [
        # the reference validation mesh: one apply, all launch and latency
        {"name": "apply_f64_16_p4", "kind": "apply", "dim": 16, "degree": 4, "dtype": "f64"},
        # the headline benchmark: 26.2 M DoF, one FP64 apply
        {"name": "apply_f64_1024_p4", "kind": "apply", "dim": 1024, "degree": 4, "dtype": "f64"},
        # the high-degree end of the throughput sweep, on an odd mesh (ragged tiles)
        {"name": "apply_f64_443_p8", "kind": "apply", "dim": 443, "degree": 8, "dtype": "f64"},
        # the FP32 apply at the size of the mixed-precision benchmark
        {"name": "apply_f32_512_p6", "kind": "apply", "dim": 512, "degree": 6, "dtype": "f32"},
        # the FP32 apply of high-degree solves (degrees 7 and 8 of the serving mix), odd mesh
        {"name": "apply_f32_391_p7", "kind": "apply", "dim": 391, "degree": 7, "dtype": "f32"},
        # the headline apply for a caller whose vectors live in (page-locked) host memory
        {"name": "apply_host_1024_p4", "kind": "apply_host", "dim": 1024, "degree": 4},
        # the right-hand side that every solve of the serving mix starts from
        {"name": "rhs_512_p6", "kind": "rhs", "dim": 512, "degree": 6},
        # the reference validation solve: 16 x 16, p = 4, CG to 1e-12
        {"name": "cg_f64_16_p4", "kind": "cg", "dim": 16, "degree": 4, "tol": 1e-12},
        # a large plain FP64 solve: hundreds of iterations over vectors of 25 MB
        {"name": "cg_f64_256_p6", "kind": "cg", "dim": 256, "degree": 6, "tol": 1e-10},
        # the mixed-precision benchmark, to a true relative residual of 1e-10
        {"name": "mixed_512_p6", "kind": "mixed", "dim": 512, "degree": 6, "tol": 1e-10},
        # uneven problems solved together, as in the batched benchmark (part b)
        {"name": "batch_32_uneven", "kind": "batch", "count": 32, "lo": 16, "hi": 256, "mix": 2, "tol": 1e-10},
        # a burst of the serving stream: 24 requests at once, from submission to the solutions on the host
        {"name": "serve_24", "kind": "serve", "count": 24, "lo": 8, "hi": 384, "mix": 3, "tol": 1e-10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "apply", "apply_host", "rhs", "cg", "mixed", "batch", "serve"])
    degree = rng.randint(1, 8)
    if kind in ("apply", "apply_host", "rhs"):
        # up to the headline's 26 M DoF (the right-hand side: 13 M)
        cap = int(math.sqrt((26e6 if kind == "apply" else 13e6)) / (degree + 1))
        case = {"kind": kind, "dim": _log_int(rng, 8, cap), "degree": degree}
        if kind == "apply":
            case["dtype"] = rng.choice(["f64", "f32"])
        return case
    degree = max(2, degree)
    if kind == "cg":
        dim = _log_int(rng, 8, min(300, int(2000 / (degree + 1))))
        return {"kind": kind, "dim": dim, "degree": degree, "tol": 1e-12 if dim <= 64 else 1e-10}
    if kind == "mixed":
        return {"kind": kind, "dim": _log_int(rng, 8, min(512, int(3584 / (degree + 1)))), "degree": degree, "tol": 1e-10}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 24), "lo": rng.randint(8, 32), "hi": rng.randint(48, 200),
                "mix": rng.randint(0, 1 << 20), "tol": 1e-10}
    return {"kind": kind, "count": rng.randint(2, 20), "lo": rng.randint(8, 24), "hi": rng.randint(48, 256),
            "mix": rng.randint(0, 1 << 20), "tol": 1e-10}


def _penalty(degree):
    return float(degree * degree)


def _modes(rng):
    """f = a sum of 4 modes A sin(k pi x) sin(l pi y), k, l in 1..8, A ~ N(0, 1)."""
    return ([float(a) for a in rng.normal(size=4)], [int(k) for k in rng.integers(1, 9, 4)],
            [int(k) for k in rng.integers(1, 9, 4)])


def _problems(case, seed):
    """The (dim, degree, modes) list of a batch or burst: the mix of sizes is the case's, the right-hand sides the seed's."""
    sizes = np.random.default_rng(case["mix"])
    data = np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        dim = int(round(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        out.append((dim, int(sizes.integers(2, 9)), _modes(data)))
    return out


def _vector(n, seed, dtype=torch.float64):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64).mul_(2.0).sub_(1.0).to(dtype)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        probs = _problems(case, seed)
        if kind == "serve":
            reqs = [(d, p, _penalty(p), case["tol"], sipg.Modes.make(*m)) for d, p, m in probs]
            return {"case": case, "server": sipg.Server(budget_bytes=32 << 30), "requests": reqs}
        batch = sipg.Batch([(d, p, _penalty(p)) for d, p, _ in probs])
        bs = [batch.op(i).rhs("modes", modes=sipg.Modes.make(*m)) for i, (_, _, m) in enumerate(probs)]
        return {"case": case, "batch": batch, "bs": bs}
    op = sipg.Operator(case["dim"], case["degree"], _penalty(case["degree"]))
    state = {"case": case, "op": op}
    if kind == "apply":
        # a vector of the throughput sweep: i.i.d. uniform [-1, 1]
        state["x"] = _vector(op.ndof, seed, torch.float64 if case["dtype"] == "f64" else torch.float32)
        state["y"] = torch.empty_like(state["x"])
    elif kind == "apply_host":
        state["x"] = torch.empty(op.ndof, dtype=torch.float64, pin_memory=True)
        state["x"].copy_(_vector(op.ndof, seed))
        state["y"] = torch.empty(op.ndof, dtype=torch.float64, pin_memory=True)
    else:
        modes = sipg.Modes.make(*_modes(np.random.default_rng(seed)))
        if kind == "rhs":
            state["modes"], state["b"] = modes, op.empty()
        else:
            state["b"] = op.rhs("modes", modes=modes)
    return state


def run(state):
    case = state["case"]
    kind, op = case["kind"], state.get("op")
    if kind == "apply":
        return op.apply(state["x"], out=state["y"])
    if kind == "apply_host":
        return op.apply_host(state["x"].numpy(), out=state["y"].numpy())
    if kind == "rhs":
        return op.rhs("modes", modes=state["modes"], out=state["b"])
    if kind == "cg":
        x = torch.zeros_like(state["b"])
        op.cg(x, state["b"], case["tol"], relative=True)
        return x
    if kind == "mixed":
        x = torch.zeros_like(state["b"])
        op.solve_mixed(x, state["b"], inner_tol=3e-2, outer_tol=case["tol"])
        return x
    if kind == "batch":
        xs = [torch.zeros_like(b) for b in state["bs"]]
        state["batch"].solve_mixed(xs, state["bs"], outer_tol=case["tol"])
        return xs
    server = state["server"]
    ids = [server.submit(d, p, pen, tol, modes=m)[0] for d, p, pen, tol, m in state["requests"]]
    while server.step()[0] or server.stats().queued:
        pass
    out = []
    for rid, (d, p, _, _, _) in zip(ids, state["requests"]):
        out.append(server.solution(rid, d * d * (p + 1) ** 2))
        server.release(rid)
    return out


def work(case):
    """Vectors read and written once, and the multiply-adds of one operator apply (a solve needs at least two)."""
    if case["kind"] in ("batch", "serve"):
        dofs = [(d * d * (p + 1) ** 2, p) for d, p, _ in _problems(case, 0)]
    else:
        dofs = [(case["dim"] ** 2 * (case["degree"] + 1) ** 2, case["degree"])]
    n = sum(d for d, _ in dofs)
    apply_flops = sum(2.0 * d * (2 * (p + 1) + 4) for d, p in dofs)
    kind = case["kind"]
    if kind == "apply":
        return {"bytes": 2.0 * n * (8 if case["dtype"] == "f64" else 4), "flops": apply_flops}
    if kind == "apply_host":
        return {"bytes": 16.0 * n, "flops": apply_flops}
    if kind == "rhs":
        return {"bytes": 8.0 * n, "flops": 8.0 * n}
    return {"bytes": 16.0 * n, "flops": 2.0 * apply_flops}


# ---- the same results from dense 64-bit linear algebra -----------------------
#
# On the tensor-product mesh the operator is A = A1 (x) W + W (x) A1, with A1
# the one-dimensional SIPG operator on dim elements and W the LGL weights.


def _lgl(p):
    """LGL nodes, weights and D[mode, node] of degree p (Newton on (1 - x^2) P_p')."""
    n = p + 1
    x = -np.cos(np.pi * np.arange(n) / p)
    for _ in range(100):
        L = np.zeros((n, n))
        L[:, 0], L[:, 1] = 1.0, x
        for k in range(2, n):
            L[:, k] = ((2 * k - 1) * x * L[:, k - 1] - (k - 1) * L[:, k - 2]) / k
        dx = (x * L[:, p] - L[:, p - 1]) / (n * L[:, p])
        x = x - dx
        if np.max(np.abs(dx)) < 1e-16:
            break
    x = 0.5 * (x - x[::-1])
    w = 2.0 / (p * n * L[:, p] ** 2)
    lag = np.array([np.prod([x[i] - x[j] for j in range(n) if j != i]) for i in range(n)])
    D = np.zeros((n, n))
    for i in range(n):
        for k in range(n):
            if i != k:
                D[i, k] = np.prod([x[k] - x[j] for j in range(n) if j not in (i, k)]) / lag[i]
    for k in range(n):
        D[k, k] = -np.sum(np.delete(D[:, k], k))
    return x, w, D


def _axis_operator(dim, p, pen):
    """A1 (m x m) and its weights (m), m = dim (p + 1)."""
    n = p + 1
    _, w, D = _lgl(p)
    d0, dN = D[:, 0], D[:, p]
    A = np.zeros((dim * n, dim * n))
    for e in range(dim):
        s = slice(e * n, e * n + n)
        A[s, s] += D @ np.diag(w) @ D.T
    for f in range(dim + 1):  # the face between elements f - 1 (its node p) and f (its node 0)
        jump, mean = np.zeros(dim * n), np.zeros(dim * n)
        kappa = 0.5 if 0 < f < dim else 1.0
        if f < dim:
            jump[f * n] = 1.0
            mean[f * n:f * n + n] = d0 * kappa
        if f > 0:
            jump[f * n - 1] = -1.0
            mean[(f - 1) * n:f * n] = dN * kappa
        lo, hi = max(0, (f - 1) * n), min(dim * n, (f + 1) * n)
        j, m = jump[lo:hi], mean[lo:hi]
        A[lo:hi, lo:hi] += np.outer(m, j) + np.outer(j, m) + pen * np.outer(j, j)
    return A, np.tile(w, dim)


def _to_grid(v, dim, n):
    """Node-major vector -> [x node, y node] on the tensor grid."""
    return v.reshape(n, n, dim, dim).flip(2).permute(3, 0, 2, 1).reshape(dim * n, dim * n)


def _from_grid(g, dim, n):
    return g.reshape(dim, n, dim, n).permute(1, 3, 2, 0).flip(2).reshape(-1)


def _rhs(dim, p, pen, modes):
    """The load vector and the weak Dirichlet terms, node-major."""
    n = p + 1
    xi, w, D = _lgl(p)
    delta = 1.0 / dim
    xcol = np.concatenate([[0.0], np.cumsum(np.full(dim, delta))[:-1]])
    yrow = np.add.accumulate(np.concatenate([[1.0], np.full(dim, -delta)]))[1:]
    node = (xi * 0.5 + 0.5) / dim
    X = torch.tensor((xcol[:, None] + node[None, :]).reshape(-1), device="cuda")  # [col, i1]
    Y = torch.tensor((yrow[::-1][:, None] + node[None, :]).reshape(-1), device="cuda")  # bottom-up [row, i2]
    f = torch.zeros(dim * n, dim * n, dtype=torch.float64, device="cuda")
    u = torch.zeros_like(f)
    for A, k, l in zip(*modes):
        s = A * torch.sin(k * math.pi * X)[:, None] * torch.sin(l * math.pi * Y)[None, :]
        f += s
        u += s / ((k * math.pi) ** 2 + (l * math.pi) ** 2)
    W = torch.tensor(np.tile(w, dim), device="cuda")
    b = f * (W * (0.5 / dim))[:, None] * (W * (0.5 / dim))[None, :]
    d0, dN = torch.tensor(D[:, 0].copy(), device="cuda"), torch.tensor(D[:, p].copy(), device="cuda")
    gl, gr, gd, gu = u[0] * W, u[-1] * W, u[:, 0] * W, u[:, -1] * W
    b[0] += pen * gl
    b[-1] += pen * gr
    b[:n] += d0[:, None] * gl[None, :]
    b[-n:] -= dN[:, None] * gr[None, :]
    b[:, 0] += pen * gd
    b[:, -1] += pen * gu
    b[:, :n] += gd[:, None] * d0[None, :]
    b[:, -n:] -= gu[:, None] * dN[None, :]
    return _from_grid(b, dim, n)


def _direct_solve(dim, p, pen, b):
    """A^-1 b through the eigenvectors of the axis operator."""
    n = p + 1
    A1, w = _axis_operator(dim, p, pen)
    s = torch.tensor(1.0 / np.sqrt(w), device="cuda")
    lam, Q = torch.linalg.eigh(torch.tensor(A1, device="cuda") * s[:, None] * s[None, :])
    V = s[:, None] * Q
    B = V.T @ _to_grid(b, dim, n) @ V
    return _from_grid(V @ (B / (lam[:, None] + lam[None, :])) @ V.T, dim, n)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        out = []
        for d, p, m in _problems(case, seed):
            if d * (p + 1) > EXACT_SOLVE_NODES // 4:  # the direct solves of all problems have to stay quick
                out.append(None)
                continue
            x = _direct_solve(d, p, _penalty(p), _rhs(d, p, _penalty(p), m))
            out.append(x.cpu().numpy() if kind == "serve" else x)
        return out
    dim, p = case["dim"], case["degree"]
    n, pen = p + 1, _penalty(p)
    if kind in ("apply", "apply_host"):
        x = _vector(dim * dim * n * n, seed, torch.float32 if case.get("dtype") == "f32" else torch.float64).double()
        A1, w = _axis_operator(dim, p, pen)
        A1, w = torch.tensor(A1, device="cuda"), torch.tensor(w, device="cuda")
        U = _to_grid(x, dim, n)
        y = _from_grid((A1 @ U) * w[None, :] + w[:, None] * (U @ A1.T), dim, n)
        return y.cpu().numpy() if kind == "apply_host" else y
    b = _rhs(dim, p, pen, _modes(np.random.default_rng(seed)))
    if kind == "rhs":
        return b
    return _direct_solve(dim, p, pen, b) if dim * n <= EXACT_SOLVE_NODES else None
