"""Rounding of the element pass's sums: the stiffness against FP64, beside the
no-allocation entry point's, which sums the same contractions in the order of
the reference (the local part, then the two five-term sums, each formed apart)."""
import ctypes as C

import numpy as np
import pytest

from axisem_gb300 import _abi
from axisem_gb300.mesh import random_gvec, structured_mesh
from axisem_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def _fp(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


def _rel(a, b):
    return float(np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("pole", [0, 1, 2])
def test_stiffness_rounds_as_the_sums_formed_apart(gpu_lib, orc, pole):
    """Both kernels' errors are those of the same FP32 terms, over 1e5 values and
    more: their rms differ by sampling (below 1 %) and by the order of a few
    products per point (1 %), where a chain of ten terms on top of the local
    part adds 5 %."""
    m = structured_mesh(90, 80, pole, terms="pole", axial="random1pct", seed=21)
    u = random_gvec(m, seed=22)
    ref = orc.stiffness_assembled(m, u, np.float64)
    with Solver(m) as s:
        step = _rel(s.stiffness_assembled(u), ref)
    f = np.zeros_like(u, order="F")
    assert gpu_lib.axg_stiffness_assembled_noalloc(C.byref(m.desc()), _fp(u), _fp(f)) == _abi.AXG_OK
    assert step <= 1.02 * _rel(f, ref)
