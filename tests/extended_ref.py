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


def apply(dim, p, pen, x, pivot=False):
    """(A x, S), node-major.  pivot: the zero-sum rows (stiffness, derivatives)
    over differences from the line's first value, in both."""
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

    def values(U):  # what the zero-sum rows act on
        V = U.reshape(dim, n, -1)
        return V - V[:, :1] if pivot else V

    def axis(U):  # along the first index
        d, j = values(U), jump @ U
        return (K @ d).reshape(U.shape) + mean.T @ j + jump.T @ (mean @ d.reshape(U.shape) + pen * j)

    def terms(U):
        d, j = np.abs(values(U)), np.abs(jump @ U)
        v = (np.abs(K) @ d).reshape(U.shape)
        return v + np.abs(mean).T @ j + np.abs(jump).T @ (np.abs(mean) @ d.reshape(U.shape) + abs(pen) * j)

    W = np.tile(w, dim)
    U = to_grid(x.astype(L), dim, n)
    both = lambda f: from_grid(f(U) * W[None, :] + W[:, None] * f(U.T).T, dim, n)
    return both(axis), both(terms)


def line_magnitude(dim, p, x, pivot=False):
    """For each output the larger of the largest magnitudes on its row and its
    column of the element (pivot: of the differences from the line's first value)."""
    n = p + 1
    V = x.astype(L).reshape(n, n, dim * dim)  # [i1, i2, element]
    row = np.abs(V - V[:1] if pivot else V).max(0)
    col = np.abs(V - V[:, :1] if pivot else V).max(1)
    return np.maximum(row[None, :, :], col[:, None, :]).reshape(-1)


def entry_bound(dim, p, pen, x, S, pivot=False):
    """Entry-wise error bound of the FP64 apply, from S = apply(...)[1].

    FP64 chains: 2 n + 8 roundings of at most S.  Where an element's values share
    one scale 2^s, that scale is at most 2^5 times the largest value m on the
    entry's row and column (2^6 times the largest difference), and an error of
    q = 2^-55 2^s per value (4 q from a larger neighbour) passes through rows of
    absolute sum R; the total adds 4 (1/2 + (2 NE + 2) / 2) + 2 units of at most
    2 q max R (a rounding and the dropped products of low parts, per parity
    component, and the face term's rounding)."""
    n, noe = p + 1, dim * dim
    e = np.arange(noe)
    board = np.tile(np.where((e % dim + e // dim) % 2 == 0, 1.0, -1.0), n * n)
    R = apply(dim, p, pen, board)[1]
    q = L(2) ** (-50 + (1 if pivot else 0)) * line_magnitude(dim, p, x, pivot)
    NE = (n + 1) // 2
    return (2 * n + 8) * L(2) ** -53 * S + q * (4 * R + (4 * NE + 8) * 2 * R.max())
