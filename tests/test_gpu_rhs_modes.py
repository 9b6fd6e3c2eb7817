"""The right-hand side of sine sums (tabulated per axis) against the same sums
and boundary terms in numpy, for every table width (1, 4 and 8 modes) and
partly filled ones, on meshes of one element, of one row of faces between
boundary elements, and ragged against the blocks.

Tolerance: 1e-12 of the largest entry (a handful of FP64 roundings of terms of
that size, sines included)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rhs(sipg, dim, p, pen, modes):
    n = p + 1
    xi, w = sipg.lgl_table(n)
    D = sipg.dphi_table(p).reshape(n, n)
    delta = 1.0 / dim
    xc = np.concatenate([[0.0], np.add.accumulate(np.full(dim, delta))[:-1]])
    yr = np.add.accumulate(np.concatenate([[1.0], np.full(dim, -delta)]))[1:]
    node = (xi * 0.5 + 0.5) / dim
    X = xc[None, :] + node[:, None]  # [i1, col]
    Y = yr[None, :] + node[:, None]  # [i2, row]
    f, u = np.zeros((n, n, dim, dim)), np.zeros((n, n, dim, dim))
    for A, k, l in zip(*modes):
        s = A * np.sin(k * np.pi * X)[:, None, None, :] * np.sin(l * np.pi * Y)[None, :, :, None]
        f += s
        u += s / ((k * np.pi) ** 2 + (l * np.pi) ** 2)
    q = w * 0.5 / dim
    b = q[:, None, None, None] * q[None, :, None, None] * f
    wj = w[:, None]
    gL, gR = wj * u[0, :, :, 0], wj * u[p, :, :, -1]  # [i2, row]
    gD, gU = wj * u[:, 0, -1, :], wj * u[:, p, 0, :]  # [i1, col]
    b[0, :, :, 0] += pen * gL
    b[p, :, :, -1] += pen * gR
    b[:, :, :, 0] += D[:, 0][:, None, None] * gL[None]
    b[:, :, :, -1] -= D[:, p][:, None, None] * gR[None]
    b[:, 0, -1, :] += pen * gD
    b[:, p, 0, :] += pen * gU
    b[:, :, -1, :] += D[:, 0][None, :, None] * gD[:, None]
    b[:, :, 0, :] -= D[:, p][None, :, None] * gU[:, None]
    return b.reshape(-1)


@pytest.mark.parametrize("count", [0, 1, 2, 4, 5, 8])
@pytest.mark.parametrize("p,dim", [(1, 1), (2, 2), (3, 67), (8, 13)])
def test_rhs_of_modes(sipg, p, dim, count):
    rng = np.random.default_rng(10 * p + count)
    modes = (rng.normal(size=count), rng.integers(1, 9, count), rng.integers(1, 9, count))
    op = sipg.Operator(dim, p, float(p * p))
    b = op.rhs("modes", modes=sipg.Modes.make(*modes)).cpu().numpy()
    op.close()
    ref = _rhs(sipg, dim, p, float(p * p), modes)
    assert np.max(np.abs(b - ref)) <= 1e-12 * max(np.max(np.abs(ref)), 1e-3 / dim**2)
