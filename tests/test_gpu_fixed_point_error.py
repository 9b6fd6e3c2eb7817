"""The FP64 apply's rounding error against sums in extended precision, at the
degrees whose coefficients differ most in size (1 and 2) and at the ends of the
other two scale rules.

Tolerance: 2^-52 of the result in the 2-norm -- 2^-53 for the rounding of a
result to a double, as much again for the fixed-point sums before it.  (FP64
chains of 2 n + 4 roundings stay below sqrt(2 n + 4) 2^-53.)
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = np.longdouble
DIM = 10


def _lgl(p):
    """LGL weights and D[mode, node] of degree p (Newton on (1 - x^2) P_p')."""
    n = p + 1
    x = -np.cos(np.pi * np.arange(n) / p).astype(L)
    for _ in range(60):
        P = np.ones((n, n), L)
        P[:, 1] = x
        for k in range(2, n):
            P[:, k] = ((2 * k - 1) * x * P[:, k - 1] - (k - 1) * P[:, k - 2]) / L(k)
        x = x - (x * P[:, p] - P[:, p - 1]) / (n * P[:, p])
    x = (x - x[::-1]) / 2
    D = np.zeros((n, n), L)
    for i in range(n):
        for k in range(n):
            if i != k:
                num = np.prod([x[k] - x[j] for j in range(n) if j not in (i, k)] or [L(1)])
                D[i, k] = num / np.prod([x[i] - x[j] for j in range(n) if j != i])
    for k in range(n):
        D[k, k] = -np.sum(np.delete(D[:, k], k))
    return L(2) / (p * n * P[:, p] ** 2), D


def _apply(dim, p, pen, x):
    """A x as the tensor product of one axis' operator with the weights."""
    n = p + 1
    w, D = _lgl(p)
    A = np.zeros((dim * n, dim * n), L)
    for e in range(dim):
        s = slice(e * n, e * n + n)
        A[s, s] += (D * w) @ D.T
    for f in range(dim + 1):
        jump, mean = np.zeros(dim * n, L), np.zeros(dim * n, L)
        kappa = L(0.5) if 0 < f < dim else L(1)
        if f < dim:
            jump[f * n] = 1
            mean[f * n:f * n + n] = D[:, 0] * kappa
        if f > 0:
            jump[f * n - 1] = -1
            mean[(f - 1) * n:f * n] = D[:, p] * kappa
        A += np.outer(mean, jump) + np.outer(jump, mean) + L(pen) * np.outer(jump, jump)
    W = np.tile(w, dim)
    U = x.astype(L).reshape(n, n, dim, dim)[:, :, ::-1].transpose(3, 0, 2, 1).reshape(dim * n, dim * n)
    Y = (A @ U) * W + W[:, None] * (U @ A.T)
    return Y.reshape(dim, n, dim, n).transpose(1, 3, 2, 0)[:, :, ::-1].reshape(-1)


@pytest.mark.parametrize("p", [1, 2, 3, 8])
@pytest.mark.parametrize("kind", ["uniform", "normal", "signs"])
def test_error_against_extended_precision(sipg, p, kind):
    import torch

    rng = np.random.default_rng(p)
    N, noe = DIM * DIM * (p + 1) ** 2, DIM * DIM
    if kind == "signs":  # the largest sums: full magnitudes, neighbours just within the scale's room
        e = np.arange(N) % noe
        x = rng.choice([-1.0, 1.0], N) * np.where((e % DIM + e // DIM) % 2 == 1, 3.9999, 0.50001)
    else:
        x = rng.uniform(-1, 1, N) if kind == "uniform" else rng.standard_normal(N)
    op = sipg.Operator(DIM, p, float(p * p))
    y = op.apply(torch.from_numpy(x).cuda()).cpu().numpy()
    op.close()
    ref = _apply(DIM, p, p * p, x)
    d = y.astype(L) - ref
    assert np.sqrt((d * d).sum() / (ref * ref).sum()) <= 2.0 ** -52
