"""The extended-precision reference of the accuracy tests against its definition
on one element of degree 2."""
import numpy as np

import extended_ref as ext


def test_extended_reference_on_one_element():
    x = np.arange(9.0)
    _, w, D = ext.lgl(2)
    ref, S = ext.apply(1, 2, 4.0, x)
    U = x.reshape(3, 3)  # [i1, i2]
    d0, dN, e0, eN = D[:, 0], D[:, 2], np.eye(3)[0], np.eye(3)[2]
    A = (D * w) @ D.T + np.outer(d0, e0) + np.outer(e0, d0) - np.outer(dN, eN) - np.outer(eN, dN)
    A = A + 4.0 * (np.outer(e0, e0) + np.outer(eN, eN))
    expect = A @ U * w + w[:, None] * (U @ A.T)
    assert np.allclose(expect.reshape(-1).astype(float), ref.astype(float), rtol=1e-14, atol=1e-14)
    assert (S >= np.abs(ref)).all()


def test_extended_reference_matches_the_oracle(oracle):
    rng = np.random.default_rng(0)
    for p, dim in ((1, 3), (3, 2), (8, 4)):
        x = rng.uniform(-1, 1, dim * dim * (p + 1) ** 2)
        ref, S = ext.apply(dim, p, 7.0 * p, x)
        assert np.max(np.abs(ext.apply(dim, p, 7.0 * p, x, pivot=True)[0] - ref) / S) <= 1e-17
        assert np.max(np.abs(oracle.apply(p, dim, 7.0 * p, x) - ref) / S) <= (2 * p + 8) * 2.0 ** -53
