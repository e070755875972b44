"""The debug build with device bounds checks (-DAXG_DEVICE_CHECKS) compiles, links
and loads: its record of a violation exists once per translation unit of kernels."""
import ctypes as C

from axisem_gb300 import _abi


def test_checked_build_links(tmp_path, monkeypatch):
    import axisem_gb300.build as b
    monkeypatch.setattr(b, "OUT", tmp_path)
    monkeypatch.setattr(b, "LIB", tmp_path / b.LIB.name)
    lib = C.CDLL(str(b.build(force=True, extra=["-DAXG_DEVICE_CHECKS"])))
    out = (C.c_int32 * 8)()
    assert lib.axg_device_check_report(out) != _abi.AXG_ERR_UNSUPPORTED
