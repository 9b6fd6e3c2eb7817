"""The FP64 apply on vectors whose values differ widely inside an element or
between neighbours: entry by entry within the bound of FP64 chains where one
scale does not fit an element (extended_ref.entry_bound says where that is), and
the same bits from every tile shape, NaN, infinity and denormals included."""
import ctypes as C

import numpy as np
import pytest

import extended_ref as ext

pytestmark = pytest.mark.gpu

KINDS = ("node2^4", "node2^13", "node2^50", "graded1e-14", "graded1e-20", "scales", "impulse", "sparse", "half")


def vector(kind, p, dim, rng):
    n, noe = p + 1, dim * dim
    x = rng.uniform(-1, 1, n * n * noe)
    V = x.reshape(n * n, noe)
    k = (n // 2) * n + n // 2
    if kind.startswith("node"):  # one node of each element scaled up
        V[k] *= 2.0 ** int(kind[6:])
    elif kind.startswith("graded"):  # one node at 1, the rest far below
        V *= float(kind[6:])
        V[k, ::2] = 1.0
        V[0, 1::2] = 1.0
    elif kind == "scales":  # neighbouring elements up to 16 decades apart
        V *= 10.0 ** rng.integers(-8, 8, noe)
    elif kind == "impulse":
        V[:] = 0.0
        V[k, noe // 2] = -3.0
    elif kind == "sparse":
        V *= rng.random(V.shape) < 0.02
    elif kind == "half":  # zero on one side of a line through the mesh
        V[:, np.arange(noe) % dim > dim // 2] = 0.0
    elif kind == "spike":  # equal values but for the first node's
        V[:] = 1e8
        V[0] = 0.0
    return x


def shapes(op, p):
    yield lambda: op.set_tile("f64", 4)
    yield lambda: op.set_tile("f64", 2)
    if p <= 7:
        yield lambda: op.set_tile("f64", 8)
    yield lambda: op.set_pernode(0)
    yield lambda: op.set_pernode(1)


@pytest.mark.parametrize("p,dim", [(1, 9), (2, 9), (3, 7), (4, 35), (5, 6), (6, 10), (7, 5), (8, 9)])
@pytest.mark.parametrize("factor", [1.0, 100.0])
def test_entrywise_error(sipg, p, dim, factor):
    import torch

    rng = np.random.default_rng(p)
    pen = p * p * factor
    op = sipg.Operator(dim, p, pen)
    for kind in KINDS:
        x = vector(kind, p, dim, rng)
        ref, S = ext.apply(dim, p, pen, x)
        bound = ext.entry_bound(dim, p, pen, x, S)
        xt, first = torch.from_numpy(x).cuda(), None
        for choose in shapes(op, p):
            choose()
            y = op.apply(xt)
            if first is None:
                first = y
                over = np.abs(y.cpu().numpy() - ref) - bound
                assert over.max() <= 0, (kind, int(over.argmax()), float(over.max()))
            else:
                assert torch.equal(y, first), kind
    op.close()


@pytest.mark.parametrize("p,dim", [(1, 40), (2, 33), (4, 35), (5, 37), (6, 33), (8, 34)])
def test_shapes_agree_without_a_scale(sipg, p, dim):
    """NaN, infinity, denormals and the ends of the exponent range: the same bits
    from every tile shape, and the elements that do not touch one keep theirs."""
    import torch

    rng = np.random.default_rng(p)
    n, noe = p + 1, dim * dim
    op = sipg.Operator(dim, p, float(p * p))
    clean = rng.uniform(-1, 1, n * n * noe)
    for value in (np.nan, np.inf, -np.inf, 1e300, 5e-324, 1e-300):
        x = clean.copy()
        V = x.reshape(n * n, dim, dim)
        row, col = dim // 2, dim // 3
        if abs(value) < 1.0:  # elements with nothing larger
            V[:, row, col] = 0.0
        V[n + n // 2, row, col] = value
        first = base = None
        for choose in shapes(op, p):
            choose()
            y = op.apply(torch.from_numpy(x).cuda()).view(torch.int64)
            if first is None:
                first = y
                base = op.apply(torch.from_numpy(clean).cuda()).view(torch.int64).view(-1, dim, dim)
                away = torch.ones(dim, dim, dtype=torch.bool, device="cuda")
                for r, c in ((row, col), (row - 1, col), (row + 1, col), (row, col - 1), (row, col + 1)):
                    away[r, c] = False
                assert torch.equal(y.view(-1, dim, dim)[:, away], base[:, away]), value
            else:
                assert torch.equal(y, first), value
    op.close()


@pytest.mark.parametrize("p,dim", [(1, 9), (2, 9), (3, 7), (4, 35), (5, 6), (6, 10), (7, 5), (8, 9)])
@pytest.mark.parametrize("factor", [1.0, 100.0])
def test_residual_entrywise_error(sipg, p, dim, factor):
    """The residual evaluation over differences (-A x for b = 0), per entry."""
    import torch

    rng = np.random.default_rng(10 + p)
    pen = p * p * factor
    op = sipg.Operator(dim, p, pen)
    b, r, rel = op.empty().zero_(), op.empty(), C.c_double()
    for kind in KINDS + ("spike",):
        x = vector(kind, p, dim, rng)
        ref, S = ext.apply(dim, p, pen, x, pivot=True)
        bound = ext.entry_bound(dim, p, pen, x, S, pivot=True)
        xt, first = torch.from_numpy(x).cuda(), None
        for rows in (4, 2, 8) if p <= 7 else (4, 2):
            op.set_tile("f64", rows)
            st = sipg.lib().sipg_residual_f64(op._h, xt.data_ptr(), b.data_ptr(), r.data_ptr(), C.byref(rel),
                                              torch.cuda.current_stream().cuda_stream)
            assert st == 0
            if first is None:
                first = r.clone()
                over = np.abs(-r.cpu().numpy() - ref) - bound
                assert over.max() <= 0, (kind, int(over.argmax()), float(over.max()))
                norm = float(np.sqrt((ref * ref).sum()))
                assert abs(rel.value - norm) <= 1e-12 * norm
            else:
                assert torch.equal(r, first), kind
    op.close()
