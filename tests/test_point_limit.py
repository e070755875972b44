"""Element blocks hold a point's number in 28 bits: the planner, which every solve
and both domains go through, refuses a mesh of more points."""
import ctypes as C

import pytest

from axisem_gb300 import _abi
from axisem_gb300.mesh import coupled_mesh


@pytest.mark.parametrize("field", ["nglob_solid", "nglob_fluid"])
def test_more_than_28_bits_of_points_are_refused(lib, field):
    d = coupled_mesh(4, 3, 2, 2).desc()
    info = _abi.Info()
    assert lib.axg_plan_check(C.byref(d), 0, -1, C.byref(info)) == _abi.AXG_OK
    setattr(d, field, 1 << 28)
    assert lib.axg_plan_check(C.byref(d), 0, -1, C.byref(info)) == _abi.AXG_ERR_BAD_DESC
    assert "nglob" in lib.axg_last_error(None).decode()
