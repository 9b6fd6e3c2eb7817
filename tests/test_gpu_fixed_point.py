"""The FP64 apply's fixed-point sums (sipg_fx.cuh) where they could go wrong:
element scales far apart, single and scattered non-zeros, magnitudes at the ends
of the exponent range, large and zero penalties, and values without a scale
(NaN, infinity), which send their tile to the plain FP64 code -- at degrees
with and without a middle node, on meshes that fill no tile, one tile and
ragged tiles, with the element and the per-node tiles.

Tolerance: the FP64 bar of the apply tests, 1e-12 of the largest entry (a value's
quantum is 2^-55 of its element's largest, so sums of 2 n + 4 terms stay far
below it).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL64 = 1e-12
CASES = [(1, 5), (2, 33), (3, 2), (4, 35), (5, 9), (6, 1), (7, 34), (8, 33)]


@pytest.fixture(scope="module")
def torch():
    import torch as t

    return t


def _vector(kind, p, d, rng):
    nn, noe = (p + 1) ** 2, d * d
    x = rng.uniform(-1, 1, nn * noe)
    if kind == "scales":  # neighbouring elements up to 16 decades apart
        x *= np.tile(10.0 ** rng.integers(-8, 8, noe), nn)
    elif kind == "unit":
        x[:] = 0.0
        x[(nn // 2) * noe + noe // 2] = -3.0
    elif kind == "sparse":
        x *= rng.random(x.size) < 0.02
    elif kind == "huge":
        x *= 1e280
    elif kind == "tiny":
        x *= 1e-270
    elif kind == "smooth":
        e = np.arange(nn * noe) % noe
        x = 1.0 + np.sin(3.0 * (e % d) / d) * np.cos(2.0 * (e // d) / d) + 1e-9 * x
    return x


def _shapes(sipg, op):
    yield lambda: op.set_tile("f64", 4)
    yield lambda: op.set_tile("f64", 2)
    yield lambda: op.set_pernode(0)
    yield lambda: op.set_pernode(1)


@pytest.mark.parametrize("pen_factor", [1.0, 100.0, 0.0])
@pytest.mark.parametrize("p,d", CASES)
def test_fixed_point_apply_matches_oracle(sipg, oracle, torch, p, d, pen_factor):
    rng = np.random.default_rng(1000 * p + d)
    pen = p * p * pen_factor
    op = sipg.Operator(d, p, pen)
    for kind in ("uniform", "scales", "unit", "sparse", "huge", "tiny", "smooth", "zero"):
        x = _vector(kind, p, d, rng) * (0.0 if kind == "zero" else 1.0)
        ref = oracle.apply(p, d, pen, x)
        xt, first = torch.from_numpy(x).cuda(), None
        for choose in _shapes(sipg, op):
            choose()
            y = op.apply(xt)
            if first is None:
                first = y
                err = np.max(np.abs(y.cpu().numpy() - ref))
                assert err <= RTOL64 * np.max(np.abs(ref)), (kind, err)
            elif kind != "tiny":  # every tile shape: the same integers
                assert torch.equal(y, first), kind
    op.close()


@pytest.mark.parametrize("p,d", [(2, 40), (5, 37), (8, 33)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_value_without_a_scale_stays_local(sipg, torch, p, d, bad):
    """A NaN or infinity reaches its element and the four around it, nothing
    else; the other elements' results stay those of the clean vector."""
    op = sipg.Operator(d, p, float(p * p))
    g = torch.Generator(device="cuda").manual_seed(p)
    x = torch.rand(op.ndof, device="cuda", dtype=torch.float64, generator=g) * 2 - 1
    clean = op.apply(x).view(-1, d, d)
    row, col = d // 2, d // 3
    xb = x.clone().view(-1, d, d)
    xb[(p + 1) ** 2 // 2, row, col] = bad
    for choose in _shapes(sipg, op):
        choose()
        y = op.apply(xb.view(-1)).view(-1, d, d)
        assert not torch.isfinite(y[:, row, col]).all()
        touched = torch.zeros(d, d, dtype=torch.bool, device="cuda")
        for r, c in ((row, col), (row - 1, col), (row + 1, col), (row, col - 1), (row, col + 1)):
            touched[r, c] = True
        diff = (y - clean)[:, ~touched].abs().max().item()
        assert diff <= RTOL64 * clean.abs().max().item()
    op.close()

