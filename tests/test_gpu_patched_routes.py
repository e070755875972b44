"""GPU tests of routes that few meshes take: patched solids (more than 131 072
elements) in batches, with attenuation at every GLL point and in compensated
symplectic runs; more solves of a kernel class than a launch takes; absorbing
solves, whose fluid points are finished in a launch of their own, beside others.

Batches are bit for bit each solve's own run.  Against the FP64 oracle: relative
L2 <= 1e-4 after a few steps, the bar of the other parity tests."""
import numpy as np
import pytest

from axisem_gb300 import _abi
from axisem_gb300.mesh import add_attenuation, coupled_mesh, gauss_at, gvec_to_elemental, random_gvec
from axisem_gb300.solver import Batch, Solver, symplectic_coefficients

pytestmark = pytest.mark.gpu

PATCHED = (367, 359, 9)   # not multiples of a patch's 8 x 8
FIELDS = (_abi.FIELD_DISP, _abi.FIELD_VELO, _abi.FIELD_ACC0, _abi.FIELD_CHI, _abi.FIELD_DCHI, _abi.FIELD_DDCHI0)
N = 13   # a graph of eight steps and single ones


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


def _mesh(size, pole, **kw):
    return coupled_mesh(*size, pole, niter=N, num_rec=4, seis_it=1, terms="pole", **kw)


def _start(m, comp, seed, share=None):
    s = Solver(m, share_with=share)
    s.set_compensated(comp)
    u = random_gvec(m, seed=seed)
    if m.src_type == 0:
        u[:, 1] = 0.0
    s.upload_disp(u)
    return s


def _result(s):
    return [s.receivers()] + [s.get_state(f) for f in FIELDS]


def _batch_equals_alone(specs, share=False):
    """specs: (mesh, compensated, seed of the initial displacement)"""
    alone = []
    for m, comp, seed in specs:
        with _start(m, comp, seed) as s:
            s.run(1, N)
            alone.append(_result(s))
    solvers = []
    try:
        for m, comp, seed in specs:
            solvers.append(_start(m, comp, seed, share=solvers[0] if share and solvers else None))
        with Batch(solvers) as b:
            b.run([1] * len(solvers), N)
        for s, want in zip(solvers, alone):
            assert np.abs(want[1]).max() > 0
            for a, w in zip(_result(s), want):
                assert np.array_equal(a, w)
    finally:
        for s in reversed(solvers):
            s.close()


@pytest.mark.parametrize("pole,comp", [(0, False), (1, True), (2, False), (2, True)])
def test_patched_solid_in_a_batch(gpu_lib, pole, comp):
    big, small = _mesh(PATCHED, pole, src_row=11), _mesh((31, 17, 5), pole, src_row=4)
    _batch_equals_alone([(big, comp, 5), (small, comp, 6), (small, not comp, 7)])


def test_two_patched_solids_of_a_class(gpu_lib):
    _batch_equals_alone([(_mesh(PATCHED, 1, src_row=8), False, 5), (_mesh((401, 331, 6), 1, src_row=7), False, 6)])


def test_more_solves_than_a_launch_takes(gpu_lib):
    m = _mesh((19, 11, 4), 1, src_row=4)
    _batch_equals_alone([(m, False, seed) for seed in range(14)], share=True)


@pytest.mark.parametrize("order", [(False, True), (True, False), (True, True, False)])
def test_absorbing_solves_beside_others(gpu_lib, order):
    specs = [(_mesh((31 + 2 * k, 17, 5), 2, src_row=4, absorbing=a), False, 5 + k) for k, a in enumerate(order)]
    _batch_equals_alone(specs)


def _against_oracle(orc, m, n, scheme=None, comp=False):
    u = random_gvec(m, seed=5)
    if m.src_type == 0:
        u[:, 1] = 0.0
    t = orc.TimeLoop(m, np.float64)
    t.disp[...] = gvec_to_elemental(m, u)
    comps = [0, 2] if m.src_type == 0 else [0, 1, 2]
    with Solver(m) as s:
        s.set_compensated(comp)
        if scheme is not None:
            _, _, coeff = symplectic_coefficients(scheme, m.deltat)
            stf = gauss_at(np.arange(m.niter)[:, None] * m.deltat + coeff[None, :], 20 * m.deltat)
            s.set_time_scheme(scheme, stf)
            assert t.run_symplectic(1, n, scheme, stf) == 0
        else:
            assert t.run(1, n) == 0
        s.upload_disp(u)
        s.run(1, n)
        assert rel(s.get_state(_abi.FIELD_DISP)[..., comps], t.disp[..., comps]) <= 1e-4
        assert rel(s.get_state(_abi.FIELD_VELO)[..., comps], t.velo[..., comps]) <= 1e-4
        assert rel(s.get_state(_abi.FIELD_CHI), t.chi) <= 1e-4
        if m.anel is not None:
            mc = [0, 1, 2, 4] if m.src_type == 0 else list(range(6))   # (the monopole never writes 4 and 6)
            assert rel(s.get_state(_abi.FIELD_MEMVAR)[:, mc], t.memvar[:, mc]) <= 1e-4


@pytest.mark.parametrize("pole", [0, 1, 2])
def test_patched_solid_attenuated_at_every_point(gpu_lib, orc, pole):
    m = add_attenuation(_mesh(PATCHED, pole, src_row=11), n_sls=2, coarse_grained=False)
    _against_oracle(orc, m, 4)


@pytest.mark.parametrize("pole", [0, 1, 2])
def test_patched_solid_compensated_symplectic(gpu_lib, orc, pole):
    _against_oracle(orc, _mesh(PATCHED, pole, src_row=11), 4, scheme=_abi.SCHEME_SYMPLEC4, comp=True)


@pytest.mark.parametrize("pole", [0, 1, 2])
@pytest.mark.parametrize("size", [(60, 50, 5), (187, 151, 5)])
def test_stiffness_call_and_step_take_the_same_form(gpu_lib, pole, size):
    """Scattered dipoles and quadrupoles whose blocks come from HBM run at three
    CTAs per SM, others at four, the stiffness call as the step."""
    with Solver(_mesh(size, pole, src_row=4)) as s:
        info = s.info()
    assert info["ctas_per_sm_force"] == info["ctas_per_sm_step"] == (3 if pole > 0 and size[0] > 100 else 4)
