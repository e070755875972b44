"""Solves whose displacement blows up.  The guard reads the displacement that a
step forms; the reference completes that step and stops before the next one
(runtime_info, SOLVER/time_evol_wave.F90:998-1056).  The step is the same bits as
without the guard, and the steps queued behind it do nothing."""
import ctypes as C
import re
import time

import numpy as np
import pytest

from axisem_gb300 import _abi
from axisem_gb300.mesh import add_attenuation, coupled_mesh, gauss_at, random_gvec
from axisem_gb300.solver import AxgError, Batch, Solver, symplectic_coefficients

pytestmark = pytest.mark.gpu

SMALL, PATCHED = (37, 23, 7), (367, 359, 5)   # scattered; patched
NITER = 48


def _mesh(size, pole, mode, magnitude=1e20, deltat=2e-6):
    m = coupled_mesh(*size, pole, niter=NITER, num_rec=3, seis_it=1, terms="pole", src_row=8, deltat=deltat,
                     absorbing=mode == "absorb")
    if mode in ("cg4", "full"):
        add_attenuation(m, coarse_grained=mode == "cg4")
    m.magnitude = magnitude
    return m


def _solver(m, mode, u=None):
    s = Solver(m)
    s.set_compensated(mode == "comp")
    if mode == "symplec4":
        _, _, coeff = symplectic_coefficients(_abi.SCHEME_SYMPLEC4, m.deltat)
        s.set_time_scheme(_abi.SCHEME_SYMPLEC4,
                          gauss_at(np.arange(m.niter)[:, None] * m.deltat + coeff[None, :], 20 * m.deltat))
    if u is not None:
        s.upload_disp(u)
    return s


def _state(s, mode):
    fields = [_abi.FIELD_DISP, _abi.FIELD_VELO, _abi.FIELD_ACC0, _abi.FIELD_CHI, _abi.FIELD_DCHI, _abi.FIELD_DDCHI0]
    if mode in ("cg4", "full"):
        fields += [_abi.FIELD_MEMVAR, _abi.FIELD_ATT_SRC_TR, _abi.FIELD_ATT_SRC_DEV]
    if mode == "comp":
        fields += [_abi.FIELD_DISP_COMP, _abi.FIELD_VELO_COMP, _abi.FIELD_CHI_COMP, _abi.FIELD_DCHI_COMP]
    return {f: s.get_state(f) for f in fields}


def _blown(call):
    """The iteration whose displacement blew up."""
    with pytest.raises(AxgError) as ei:
        call()
    assert ei.value.code == _abi.AXG_ERR_BLOWUP
    return int(re.search(r"time step (\d+)", str(ei.value)).group(1)) - 1


CASES = [(SMALL, 0, "plain", None), (SMALL, 0, "plain", 5), (SMALL, 1, "cg4", 5), (SMALL, 1, "cg4", None),
         (SMALL, 2, "comp", 5), (SMALL, 1, "full", 5), (SMALL, 1, "absorb", 5), (SMALL, 2, "symplec4", 5),
         (PATCHED, 2, "plain", 5), (PATCHED, 2, "plain", None), (PATCHED, 1, "comp", 5), (PATCHED, 0, "symplec4", 5)]


@pytest.mark.parametrize("size,pole,mode,seed", CASES)
def test_step_that_blows_up_is_completed(gpu_lib, size, pole, mode, seed):
    """From a random displacement (the first step) and from the source (a later
    one): the state is that of the same steps without the guard."""
    m = _mesh(size, pole, mode, 1e-20)
    u = None if seed is None else random_gvec(m, seed=seed)
    if u is not None and pole == 0:
        u[:, 1] = 0.0
    with _solver(m, mode, u) as s:
        k = _blown(lambda: s.run(1, NITER))
    assert 1 <= k < NITER and (k == 1) == (seed is not None)
    with _solver(m, mode, u) as s:
        assert _blown(lambda: s.run(1, k)) == k
        got = _state(s, mode)
    with _solver(_mesh(size, pole, mode), mode, u) as s:
        s.run(1, k)
        want = _state(s, mode)
    assert np.abs(want[_abi.FIELD_VELO]).max() > 0
    for f in want:
        assert np.array_equal(got[f], want[f]), f


@pytest.mark.parametrize("size,pole,mode", [((360, 350, 5), 1, "cg4"), ((360, 350, 5), 2, "plain"), (PATCHED, 2, "comp")])
def test_steps_after_a_blowup_cost_little(gpu_lib, size, pole, mode):
    """Queued steps of a stopped solve take less than half of a running one's
    (some read a few rows and states before they know)."""
    took = []
    for magnitude in (1e20, 1e-20):
        m = _mesh(size, pole, mode, magnitude, deltat=1e-7)   # (well below the mesh's limit)
        with _solver(m, mode, random_gvec(m, seed=5)) as s:
            best = np.inf
            for first in (1, 1, 1):
                t0 = time.perf_counter()
                s.run_async(first, NITER)
                if magnitude < 1:
                    _blown(s.wait)
                else:
                    s.wait()
                best = min(best, time.perf_counter() - t0)
            took.append(best)
    assert took[1] < 0.5 * took[0], took


@pytest.mark.parametrize("size,pole,mode,seed", [(SMALL, 0, "plain", 5), (SMALL, 0, "plain", None), (SMALL, 2, "comp", 5),
                                                 (SMALL, 1, "cg4", None), (SMALL, 1, "symplec4", 5), (PATCHED, 1, "comp", 5)])
def test_state_after_a_blowup_whatever_was_queued(gpu_lib, size, pole, mode, seed):
    """The displacement buffers trade roles every step; those of the steps queued
    behind a blow-up move nothing.  The state is that of the step that blew up,
    however many follow it and however they were queued; axg_run counts the steps
    of the graphs up to the one that stopped (16 each)."""
    m = _mesh(size, pole, mode, 1e-20)
    u = None if seed is None else random_gvec(m, seed=seed)
    if u is not None and pole == 0:
        u[:, 1] = 0.0
    with _solver(m, mode, u) as s:
        k = _blown(lambda: s.run(1, NITER))
    with _solver(_mesh(size, pole, mode), mode, u) as s:
        s.run(1, k)
        want = _state(s, mode)

    def samples(s):
        n = C.c_int32()
        out = np.zeros((s.nseismo, 3, m.num_rec), np.float32, order="F")
        assert gpu_lib.axg_get_receivers(s.h, out.ctypes.data_as(C.POINTER(C.c_float)), s.nseismo, C.byref(n)) == 0
        return n.value

    def run(s, n):
        assert _blown(lambda: s.run(1, n)) == k
        assert samples(s) == min(n, 16) + 1   # (and iteration 0)

    def run_async(s, n):
        s.run_async(1, n)
        assert _blown(s.wait) == k
        assert samples(s) == n + 1

    def in_chunks(s, n):
        s.run_async(1, n)
        s.run_async(n + 1, 3)
        assert _blown(s.wait) == k

    def batch(s, n):
        with Batch([s]) as b:
            assert _blown(lambda: b.run([1], n)) == k

    for how in (run, run_async, in_chunks, batch):
        for n in (k, k + 1, 16, 17, 24, 33):
            with _solver(m, mode, u) as s:
                how(s, n)
                got = _state(s, mode)
            for f in want:
                assert np.array_equal(got[f], want[f]), (how.__name__, n, f)
