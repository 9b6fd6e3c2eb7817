"""The operator in extended precision (np.longdouble), as the tensor product of
one axis' operator with the LGL weights, and for each output the sum S of its
terms' magnitudes: what an FP64 evaluation in any order rounds at.  A face's
jump enters S after the subtraction (two equal traces give an exact zero)."""
import numpy as np

L = np.longdouble


def lgl(p):
    """LGL nodes, weights and D[mode, node] of degree p (Newton on (1 - x^2) P_p')."""
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
    return x, L(2) / (p * n * P[:, p] ** 2), D


def to_grid(x, dim, n):
    """Node-major vector -> [x node, y node] on the tensor grid."""
    return x.reshape(n, n, dim, dim)[:, :, ::-1].transpose(3, 0, 2, 1).reshape(dim * n, dim * n)


def from_grid(g, dim, n):
    return g.reshape(dim, n, dim, n).transpose(1, 3, 2, 0)[:, :, ::-1].reshape(-1)


def apply(dim, p, pen, x):
    """(A x, S), node-major."""
    n = p + 1
    _, w, D = lgl(p)
    K = (D * w) @ D.T
    jump, mean = np.zeros((dim + 1, dim * n), L), np.zeros((dim + 1, dim * n), L)
    for f in range(dim + 1):
        kappa = L(0.5) if 0 < f < dim else L(1)
        if f < dim:
            jump[f, f * n] = 1
            mean[f, f * n:f * n + n] = D[:, 0] * kappa
        if f > 0:
            jump[f, f * n - 1] = -1
            mean[f, (f - 1) * n:f * n] = D[:, p] * kappa
    pen = L(pen)

    def axis(U):  # along the first index
        v = (K @ U.reshape(dim, n, -1)).reshape(U.shape)
        j = jump @ U
        return v + mean.T @ j + jump.T @ (mean @ U + pen * j)

    def terms(U):
        a = np.abs(U)
        v = (np.abs(K) @ a.reshape(dim, n, -1)).reshape(U.shape)
        j = np.abs(jump @ U)
        return v + np.abs(mean).T @ j + np.abs(jump).T @ (np.abs(mean) @ a + abs(pen) * j)

    W = np.tile(w, dim)
    U = to_grid(x.astype(L), dim, n)
    both = lambda f: from_grid(f(U) * W[None, :] + W[:, None] * f(U.T).T, dim, n)
    return both(axis), both(terms)
