"""The elimination of a front on the tensor cores (csrc/vefem_split.cuh): one front
of given entries, its inverse and solution by their residuals, and one front of p pivots and q boundary unknowns whose pivot block is the
identity, so that it is D - C B with the entries given, against the same in
extended precision, at sizes around the tile (128 x 48), the stage (32), the
exact sum (128)."""
import ctypes as ct

import numpy as np
import pytest
import torch

from ve_flow_around_cylinder_fortran_gb300 import build as B
from ve_flow_around_cylinder_fortran_gb300 import vefem as V

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    B.build()
    V.load()


def _eliminate(A, C, X, D):
    """The front [A X; C D] after its p pivots: [A^-1, A^-1 X; C, D - C A^-1 X]."""
    q, p = C.shape
    n = np.array([p + q, q], np.int32)
    ld = (n + 3) // 4 * 4
    off = np.concatenate([[0], np.cumsum(n.astype(np.int64) * ld)])
    ids = np.concatenate([np.arange(p + q), np.arange(p, p + q)]).astype(np.int64)
    idx_off = np.array([0, p + q, p + 2 * q], np.int64)
    src = np.full((2, p + 2 * q), -1, np.int32)
    src[0, p + q:] = p + np.arange(q)
    h = ct.c_void_p()
    ptr = lambda a: a.ctypes.data_as(ct.c_void_p)
    lib = V.load()
    piv = np.array([p, q], np.int32)
    child = np.array([[-1, -1], [0, -1]], np.int32)
    lev = np.array([0, 1, 2], np.int32)
    assert lib.vefem_tree_create(0, 2, 2, ptr(lev), ptr(off), ptr(n), ptr(piv), ptr(ld), ptr(child), ptr(ids),
                                 ptr(idx_off), ptr(src), ct.c_int64(p + q), ct.byref(h)) == 0
    M = np.block([[A, X], [C, D]])
    dest = (np.arange(p + q)[:, None] * int(ld[0]) + np.arange(p + q)).ravel()
    vals = torch.from_numpy(M.ravel()).cuda()
    dest = torch.from_numpy(dest.astype(np.int64)).cuda()
    buf = torch.empty(int(off[-1]), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    mp = ct.c_double()
    # the root, D - C B itself, need not be a matrix that eliminates
    lib.vefem_tree_factor(h, ct.c_void_p(vals.data_ptr()), ct.c_void_p(dest.data_ptr()), ct.c_int64(vals.numel()),
                          ct.c_void_p(buf.data_ptr()), ct.c_int64(buf.numel()), ct.c_void_p(0), ct.c_double(1e-12),
                          ct.byref(mp))
    torch.cuda.synchronize()
    got = buf[:int(off[1])].cpu().numpy().reshape(p + q, int(ld[0]))[:, :p + q]
    lib.vefem_tree_destroy(h)
    return got


def _schur(C, X, D):
    p = C.shape[1]
    return _eliminate(np.eye(p), C, X, D)[p:, p:]


def _operands(p, q, seed):
    r = np.random.default_rng(seed)
    return r.uniform(-1, 1, (q, p)), r.uniform(-1, 1, (p, q)), r.uniform(-1, 1, (q, q))


SIZES = [(1, 5), (31, 49), (32, 1), (33, 48), (47, 65), (64, 127), (96, 128), (128, 129), (129, 193), (160, 40), (300, 257)]


@pytest.mark.parametrize("p,q", SIZES)
def test_product_error(p, q):
    C, X, D = _operands(p, q, p)
    P = C.astype(np.longdouble) @ X.astype(np.longdouble)
    err = np.abs(_schur(C, X, D) - (D - P)).astype(float)
    # the rounding of the product and of the subtraction; the digits left out (below 2^-57 per k)
    S = np.abs(D - P).astype(float)
    assert np.all(err <= 2.0 ** -53 * (S + np.abs(P).astype(float)) * 1.001 + p * 2.0 ** -57)


@pytest.mark.parametrize("p,q", [(40, 70), (200, 130)])
def test_units_cost_no_digits(p, q):
    C, X, D = _operands(p, q, p)
    r = np.random.default_rng(q)
    row, col, inner = (2.0 ** r.integers(-150, 151, m) for m in (q, q, p))
    C, X, D = row[:, None] * C * inner, X * col / inner[:, None], row[:, None] * D * col
    exact = D - C.astype(np.longdouble) @ X.astype(np.longdouble)
    err = np.abs(_schur(C, X, D) - exact).astype(float)
    assert np.all(err <= 2.0 ** -53 * (p + 2) * (np.abs(C) @ np.abs(X) + np.abs(D)))


@pytest.mark.parametrize("p,q", [(1, 3), (15, 20), (16, 31), (17, 33), (31, 97), (32, 96), (33, 15), (64, 64), (97, 31),
                                 (128, 16), (129, 47), (161, 200)])
def test_inverse_and_solution(p, q):
    r = np.random.default_rng(p)
    C, X, D = _operands(p, q, q)
    scale = 2.0 ** r.integers(-40, 41, p)                # equations and unknowns of any unit
    A = (r.uniform(-1, 1, (p, p)) + 2.0 * p * np.eye(p)) * scale / scale[::-1, None]
    X = X / scale[::-1, None]
    M = _eliminate(A, C, X, D).astype(np.longdouble)
    inv, sol = M[:p, :p], M[:p, p:]
    # diagonally dominant up to its scaling: no growth, at most 2 p roundings of |A| |A^-1| per entry
    bound = lambda Y: 2.0 ** -53 * 4 * (p + 2) * (np.abs(A) @ np.abs(Y))
    assert np.all(np.abs(A @ inv - np.eye(p)) <= bound(inv))
    assert np.all(np.abs(A @ sol - X) <= bound(sol))


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_not_finite(bad):
    p, q = 50, 140
    C, X, D = _operands(p, q, 1)
    C[7, 3] = bad
    C[9] = 0.0
    got = _schur(C, X, D)
    assert not np.isfinite(got[7]).any()
    keep = np.arange(q) != 7
    assert np.array_equal(got[9], D[9])
    err = np.abs(got[keep] - (D - C.astype(np.longdouble) @ X.astype(np.longdouble))[keep]).astype(float)
    assert np.all(err <= 2.0 ** -53 * (p + 2) * (np.abs(C) @ np.abs(X) + np.abs(D))[keep])
    X[20, 90] = bad
    got = _schur(C, X, D)
    assert not np.isfinite(got[keep, 90]).any()
