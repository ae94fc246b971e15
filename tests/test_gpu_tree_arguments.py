"""Argument checks of the tree elimination's C entry points."""
import ctypes as ct

import numpy as np
import pytest
import torch

from ve_flow_around_cylinder_fortran_gb300 import build as B
from ve_flow_around_cylinder_fortran_gb300 import vefem as V

pytestmark = pytest.mark.gpu
ERR_ARG = 1


@pytest.fixture(scope="module", autouse=True)
def _built():
    B.build()
    V.load()


def _one_front(N):
    """A tree of a single front of N pivots."""
    ld = (N + 3) // 4 * 4
    a = dict(lev=np.array([0, 1], np.int32), off=np.array([0, N * ld], np.int64), n=np.array([N], np.int32),
             p=np.array([N], np.int32), ld=np.array([ld], np.int32), child=np.array([[-1, -1]], np.int32),
             ids=np.arange(N, dtype=np.int64), idx_off=np.array([0, N], np.int64), src=np.full((2, N), -1, np.int32))
    h = ct.c_void_p()
    ptr = {k: v.ctypes.data_as(ct.c_void_p) for k, v in a.items()}
    assert V.load().vefem_tree_create(0, 1, 1, ptr["lev"], ptr["off"], ptr["n"], ptr["p"], ptr["ld"], ptr["child"],
                                      ptr["ids"], ptr["idx_off"], ptr["src"], ct.c_int64(N), ct.byref(h)) == 0
    return h, N * ld


@pytest.mark.parametrize("short", [1, 100, None])
def test_short_buffer_is_refused(short):
    N = 50
    h, need = _one_front(N)
    lib = V.load()
    vals = torch.ones(N, dtype=torch.float64, device="cuda")
    dest = torch.arange(N, device="cuda") * (need // N + 1)                  # the diagonal
    buf = torch.full((need,), 7.0, dtype=torch.float64, device="cuda")       # long enough, whatever is said of it
    mp = ct.c_double()

    def factor(length):
        return lib.vefem_tree_factor(h, ct.c_void_p(vals.data_ptr()), ct.c_void_p(dest.data_ptr()), ct.c_int64(N),
                                     ct.c_void_p(buf.data_ptr()), ct.c_int64(length), ct.c_void_p(0),
                                     ct.c_double(1e-12), ct.byref(mp))

    torch.cuda.synchronize()
    assert factor(-1 if short is None else need - short) == ERR_ARG
    assert bool((buf == 7.0).all())
    assert factor(need) == 0
    lib.vefem_tree_destroy(h)


def test_handles_of_different_sizes():
    """Fronts beyond 48 KB of staged vector: the smaller handle's creation does
    not lower what the larger one's sweeps may take."""
    lib = V.load()
    N = 7000
    big, need = _one_front(N)
    small, _ = _one_front(6400)
    buf = torch.zeros(N, need // N, dtype=torch.float64, device="cuda")
    buf[torch.arange(N), torch.arange(N)] = 2.0                              # in place of an inverse
    b = torch.arange(N, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    assert lib.vefem_tree_solve(big, ct.c_void_p(buf.data_ptr()), ct.c_void_p(b.data_ptr()),
                                ct.c_void_p(x.data_ptr()), ct.c_void_p(0)) == 0
    torch.cuda.synchronize()
    assert torch.equal(x, 2.0 * b)
    lib.vefem_tree_destroy(small)
    lib.vefem_tree_destroy(big)
