"""GPU tests of the two forms of the solid's element pass: scattered (a buffer
of element contributions, summed per point) and patched (large meshes:
accumulated in shared memory, own points finished by the patch).

Sizes are where they can go wrong: solids of fewer elements than a group of
six, of group and CTA remainders, with every element on the axis; a patched
solid of ragged patches, with coupled points and the source inside patches and
on their edges.  Tolerance: relative L2 <= 1e-5 against the FP64 oracle for
the stiffness, 1e-4 for wavefields after a few steps, the bars of the other
parity tests (FP32 sums of some tens of terms in another order)."""
import numpy as np
import pytest

from axisem_gb300 import _abi, sphere
from axisem_gb300.mesh import add_attenuation, coupled_mesh, gauss_at, gvec_to_elemental, random_gvec, structured_mesh
from axisem_gb300.solver import Batch, Solver, symplectic_coefficients

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("pole", [0, 1, 2])
@pytest.mark.parametrize("ni,nj,axial", [(1, 1, "none"), (1, 1, "column"), (5, 1, "none"), (1, 7, "column"),
                                         (3, 4, "random1pct"), (5, 5, "column"), (13, 1, "random1pct")])
def test_group_remainders(gpu_lib, orc, pole, ni, nj, axial):
    m = structured_mesh(ni, nj, pole, axial=axial, seed=3)
    u = random_gvec(m, seed=4)
    with Solver(m) as s:
        f = s.stiffness_assembled(u)
        assert np.array_equal(f, s.stiffness_assembled(u))
    assert rel(f, orc.stiffness_assembled(m, u, np.float64)) <= 1e-5


@pytest.mark.parametrize("pole", [0, 1, 2])
@pytest.mark.parametrize("n_sls", [1, 5, 6, 8])
def test_memory_variables_staged(gpu_lib, orc, pole, n_sls):
    """The memory variables of up to five solids are staged in shared memory,
    further ones read directly; groups of fewer elements at the end."""
    m = add_attenuation(coupled_mesh(7, 5, 3, pole, niter=30), n_sls=n_sls)
    t = orc.TimeLoop(m, np.float64)
    assert t.run(1, m.niter) == 0
    with Solver(m) as s:
        s.run(1, m.niter)
        assert rel(s.receivers(), t.receivers()) <= 1e-4
        # (the monopole never writes components 4 and 6)
        mc = [0, 1, 2, 4] if pole == 0 else list(range(6))
        assert rel(s.get_state(_abi.FIELD_MEMVAR)[:, mc], t.memvar[:, mc]) <= 1e-4


@pytest.mark.parametrize("pole", [0, 1, 2])
def test_inner_points_of_two_elements(gpu_lib, orc, pole):
    """Inner points are summed by their place in the contributions unless a mesh
    shares one between elements: the general path for all of its points.  (The
    oracle sums edge points only; the two elements' inner forces are added here.)"""
    m = structured_mesh(7, 5, pole, axial="column", seed=6)
    u = random_gvec(m, seed=7)
    ig = m.igloc_solid.copy()
    a, b = ig[25 * 23 + 12] - 1, ig[25 * 9 + 12] - 1
    u[b] = u[a]
    want = orc.stiffness_assembled(m, u, np.float64)
    want[a] += want[b]
    want[b] = 0.0
    ig[25 * 9 + 12] = a + 1
    m.igloc_solid = ig
    with Solver(m) as s:
        f = s.stiffness_assembled(u)
    assert rel(f, want) <= 1e-5


PATCHED = (367, 359)   # 131 753 elements: patched; not multiples of a patch's 8 x 8


@pytest.mark.parametrize("pole", [0, 1, 2])
def test_patched_stiffness(gpu_lib, orc, pole):
    m = structured_mesh(*PATCHED, pole, terms="pole", axial="random1pct", seed=11)
    u = random_gvec(m, seed=12)
    with Solver(m) as s:
        f = s.stiffness_assembled(u)
        assert np.array_equal(f, s.stiffness_assembled(u))
    assert rel(f, orc.stiffness_assembled(m, u, np.float64)) <= 1e-5


@pytest.mark.parametrize("pole,comp", [(0, False), (1, False), (1, True), (2, False)])
def test_scattered_steps_from_hbm(gpu_lib, orc, pole, comp):
    """Scattered solids whose element blocks exceed what L2 keeps, with a group
    of fewer elements at the end."""
    n = 4
    m = coupled_mesh(187, 151, 5, pole, niter=n, num_rec=5, seis_it=1, terms="pole", src_row=7)
    u = random_gvec(m, seed=8)
    if pole == 0:
        u[:, 1] = 0.0
    t = orc.TimeLoop(m, np.float64)
    t.disp[...] = gvec_to_elemental(m, u)
    assert t.run(1, n) == 0
    comps = [0, 2] if pole == 0 else [0, 1, 2]
    with Solver(m) as s:
        s.set_compensated(comp)
        f = s.stiffness_assembled(u)
        assert rel(f, orc.stiffness_assembled(m, u, np.float64)) <= 1e-5
        s.upload_disp(u)
        s.run(1, n)
        assert rel(s.get_state(_abi.FIELD_DISP)[..., comps], t.disp[..., comps]) <= 1e-4
        assert rel(s.get_state(_abi.FIELD_VELO)[..., comps], t.velo[..., comps]) <= 1e-4
        assert rel(s.get_state(_abi.FIELD_CHI), t.chi) <= 1e-4


@pytest.mark.parametrize("pole,mode,absorbing", [(0, "plain", True), (1, "plain", False), (2, "comp", False),
                                                 (1, "comp", True), (2, "symplec4", False)])
def test_patched_steps(gpu_lib, orc, pole, mode, absorbing):
    """From a random displacement, so that every patch takes part."""
    n = 6
    m = coupled_mesh(PATCHED[0], PATCHED[1], 9, pole, niter=n, num_rec=9, seis_it=1, terms="pole", absorbing=absorbing,
                     src_row=8 if pole == 1 else 11)
    u = random_gvec(m, seed=5)
    if pole == 0:
        u[:, 1] = 0.0
    t = orc.TimeLoop(m, np.float64)
    t.disp[...] = gvec_to_elemental(m, u)
    with Solver(m) as s:
        s.set_compensated(mode == "comp")
        if mode == "symplec4":
            _, _, coeff = symplectic_coefficients(_abi.SCHEME_SYMPLEC4, m.deltat)
            stf = gauss_at(np.arange(n)[:, None] * m.deltat + coeff[None, :], 20 * m.deltat)
            s.set_time_scheme(_abi.SCHEME_SYMPLEC4, stf)
            assert t.run_symplectic(1, n, _abi.SCHEME_SYMPLEC4, stf) == 0
        else:
            assert t.run(1, n) == 0
        s.upload_disp(u)
        s.run(1, 4)
        s.run(5, 2)
        comps = [0, 2] if pole == 0 else [0, 1, 2]
        assert rel(s.receivers()[1:], t.receivers()[1:]) <= 1e-4
        assert rel(s.get_state(_abi.FIELD_DISP)[..., comps], t.disp[..., comps]) <= 1e-4
        assert rel(s.get_state(_abi.FIELD_VELO)[..., comps], t.velo[..., comps]) <= 1e-4
        assert rel(s.get_state(_abi.FIELD_CHI), t.chi) <= 1e-4


@pytest.mark.parametrize("seconds", [60.0, 600.0])
@pytest.mark.parametrize("pole", [0, 1, 2])
def test_mass_pairs_against_fp64_masses(gpu_lib, pole, seconds):
    """FP64 inverse masses go as FP32 pairs unless one is out of their range:
    an element held still by zero masses (pairs) against the same held by
    masses of 1e-40 (FP64 products).  The two round alike but for values within
    2^-20 of an ulp from a tie: a last bit (2^-24) here and there, over n
    steps at most n 2^-24 where every value took it each time."""
    recs = []
    for held in (0.0, 1e-40):
        m = sphere.build_mesh(50.0, sphere.SphereSolve(pole=pole, seconds=seconds))
        for name in ("inv_mass_rho_dp", "inv_mass_fluid_dp"):
            v = getattr(m, name).copy()
            v[1:4, 1:4, 40] = held
            setattr(m, name, v)
        with Solver(m) as s:
            s.set_compensated(True)
            s.run()
            recs.append((s.get_state(_abi.FIELD_DISP), s.get_state(_abi.FIELD_CHI)))
    for a, b in list(zip(*recs))[:1 if seconds < 100 else 2]:   # (the wave reaches the fluid later)
        assert np.linalg.norm(b) > 0
        assert rel(a, b) <= m.niter * 2.0 ** -24


@pytest.mark.parametrize("shared", [False, True])
def test_batch_beyond_l2(gpu_lib, shared):
    """Meshes whose blocks exceed L2 only together, with 13 steps (a graph of
    several and single ones): bit for bit each solve's own run."""
    n = 13
    ms = [coupled_mesh(110, 85, 7, p, niter=n, num_rec=4, src_row=9) for p in (1, 2)]
    ms.append(ms[1] if shared else coupled_mesh(31, 17, 5, 2, niter=n, num_rec=4, src_row=4))
    alone = []
    for m in ms:
        with Solver(m) as s:
            s.run(1, n)
            alone.append((s.receivers(), s.get_state(_abi.FIELD_DISP)))
    solvers = [Solver(m) for m in ms[:2]]
    solvers.append(Solver(ms[2], share_with=solvers[1]) if shared else Solver(ms[2]))
    with Batch(solvers) as b:
        b.run([1] * 3, n)
    for s, (rec, disp) in zip(solvers, alone):
        assert np.array_equal(s.receivers(), rec) and np.array_equal(s.get_state(_abi.FIELD_DISP), disp)
        assert np.abs(disp).max() > 0
    for s in reversed(solvers):
        s.close()
