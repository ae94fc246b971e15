"""Forward difference where its kernels hand over to each other: an element to a
CTA, four to a CTA (the last one not full), columns by field with partial runs
behind whole groups of 252 elements; clean elements, elements with a restore
residue among them and residues everywhere, against the oracle, bit for bit."""
import numpy as np
import pytest

from ve_flow_around_cylinder_fortran_gb300 import state as S
from test_gpu_fd_columns import _built, _check  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(152, 3), (457, 1), (229, 2), (153, 3), (121, 5), (607, 1), (61, 10), (63, 10), (757, 1)])
@pytest.mark.parametrize("form,nex", [("SQRT", 1), ("T", 0)])
def test_sizes(nx, ny, form, nex):
    _check(nx, ny, S.giesekus(0.1, 0.5, 0.59, form, nex=nex))


@pytest.mark.parametrize("form", ["T", "SQRT"])
@pytest.mark.parametrize("residue", [2, 40, 4000])
def test_restore_residue_with_four_elements_to_a_block(form, residue):
    _check(46, 11, S.oldroyd_b(0.5, 0.59, form, nex=1), residue=residue)
