"""The FP64 apply's rounding error with penalties well above p^2, on vectors that
are continuous across faces: the jumps are zero or tiny there, and rounding them
before the penalty multiplies them would show in the result.

Tolerance: 2^-52 of the terms' magnitudes S in the 2-norm -- 2^-53 for the
rounding of a result to a double, as much again for the sums before it.
"""
import numpy as np
import pytest

import extended_ref as ext

pytestmark = pytest.mark.gpu

DIM = 12


def _load_vector(p):
    """w_i w_j sin(2 pi x) sin(3 pi y) at the nodes: a load vector of a smooth
    function that vanishes on the boundary."""
    n, noe = p + 1, DIM * DIM
    xi, w, _ = ext.lgl(p)
    i = np.arange(n * n * noe)
    e, k = i % noe, i // noe
    x = ((e % DIM) + (xi[k // n] + 1) / 2) / DIM
    y = ((DIM - 1 - e // DIM) + (xi[k % n] + 1) / 2) / DIM
    pi = ext.L(np.pi)
    return (w[k // n] * w[k % n] * np.sin(2 * pi * x) * np.sin(3 * pi * y)).astype(np.float64)


@pytest.mark.parametrize("p", range(1, 9))
@pytest.mark.parametrize("factor", [100.0, 1e4])
def test_error_with_large_penalty(sipg, p, factor):
    import torch

    x, pen = _load_vector(p), p * p * factor
    ref, S = ext.apply(DIM, p, pen, x)
    op = sipg.Operator(DIM, p, pen)
    xt = torch.from_numpy(x).cuda()
    for choose in (lambda: op.set_pernode(0), lambda: op.set_pernode(1), lambda: op.set_tile("f64", 2),
                   lambda: op.set_tile("f64", 4)):
        choose()
        d = op.apply(xt).cpu().numpy() - ref
        assert np.sqrt((d * d).sum() / (S * S).sum()) <= 2.0 ** -52
    op.close()


