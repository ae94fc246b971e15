"""Products in digits of operands that no scaling of rows, columns or inner
indices evens: what fixed point costs there against FP64.  An entry is held to
2^-62 of the largest contribution its row (column) can make, so the error per
inner index is bounded by that, not by the product's own size."""
import numpy as np
import pytest

from test_gpu_split import _built, _schur  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,q", [(31, 49), (40, 130), (129, 100), (300, 60)])
@pytest.mark.parametrize("spread", [8, 30, 70])
def test_spread_entries(p, q, spread):
    r = np.random.default_rng(p + spread)
    C, X, D = (r.uniform(-1, 1, s) * 2.0 ** -r.uniform(0, spread, s) for s in ((q, p), (p, q), (q, q)))
    C[r.random(C.shape) < 0.1] = 0.0
    P = C.astype(np.longdouble) @ X.astype(np.longdouble)
    S = D - P
    err = np.abs(_schur(C, X, D) - S).astype(float)
    even = np.abs(X).max(axis=1)                         # the inner scaling, to a factor of 2
    row = (np.abs(C) * even).max(axis=1)
    col = (np.abs(X) / even[:, None]).max(axis=0)
    # the roundings of the product and of the subtraction, and 2^-60 per inner index, times 8
    # for the exponents that stand for the largest entries
    own = 2.0 ** -53 * 1.001 * (np.abs(S) + np.abs(P)).astype(float)
    assert np.all(err <= own + p * 2.0 ** -57 * row[:, None] * col)
    # Frobenius: no larger than an FP64 product's while entries spread over a few binades
    if spread == 8:
        fp64 = np.abs((D - C @ X) - S).astype(float)
        assert np.linalg.norm(err) <= np.linalg.norm(fp64)
