"""The 32-element FP64 tiles above the per-node tile's range: the default rows of
each degree, equal results from every number of rows, and the rounding error of
each tile, per-node ones included, for penalties on both sides of the FP64
penalty term.

Tolerance of the error: 2^-52 of the terms' magnitudes S in the 2-norm -- 2^-53
for the rounding of a result to a double, as much again for the sums before it.
"""
import numpy as np
import pytest

import extended_ref as ext

pytestmark = pytest.mark.gpu

ROWS = {1: 8, 2: 8, 3: 8, 4: 8, 5: 4, 6: 4, 7: 4, 8: 2}


@pytest.mark.parametrize("p", range(1, 9))
def test_default_rows(sipg, p):
    import torch

    dim = sipg.PERNODE_DEFAULT_DIM + 3
    op = sipg.Operator(dim, p, float(p * p))
    assert op.get_shape("f64") == (32, ROWS[p], 1)
    g = torch.Generator(device="cuda").manual_seed(p)
    x = torch.rand(op.ndof, device="cuda", dtype=torch.float64, generator=g) * 2 - 1
    first = op.apply(x)
    for rows in (2, 4, 8) if p <= 7 else (2, 4):
        op.set_tile("f64", rows)
        assert torch.equal(op.apply(x), first), rows
    op.close()


@pytest.mark.parametrize("p,dim", [(1, 9), (2, 9), (3, 7), (4, 35), (5, 6), (6, 10), (7, 5), (8, 9)])
@pytest.mark.parametrize("factor", [1.0, 100.0])
@pytest.mark.parametrize("kind", ["uniform", "smooth"])
def test_error_of_each_tile(sipg, p, dim, factor, kind):
    import torch

    n, noe = p + 1, dim * dim
    if kind == "uniform":
        x = np.random.default_rng(p).uniform(-1, 1, n * n * noe)
    else:
        xi = ((ext.lgl(p)[0] + 1) / 2).astype(np.float64)
        i = np.arange(n * n * noe)
        e, k = i % noe, i // noe
        x = np.sin(3 * (e % dim + xi[k // n]) / dim) * np.cos(2 * (dim - 1 - e // dim + xi[k % n]) / dim)
    pen = p * p * factor
    ref, S = ext.apply(dim, p, pen, x)
    op = sipg.Operator(dim, p, pen)
    xt = torch.from_numpy(x).cuda()
    choices = [lambda r=r: op.set_tile("f64", r) for r in ((2, 4, 8) if p <= 7 else (2, 4))]
    for choose in choices + [lambda: op.set_pernode(0), lambda: op.set_pernode(1)]:
        choose()
        d = op.apply(xt).cpu().numpy() - ref
        assert np.sqrt((d * d).sum() / (S * S).sum()) <= 2.0 ** -52
    op.close()
