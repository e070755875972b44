"""The compensated mode's products with FP64 inverse masses, held as FP32 pairs,
beside those of a handle that keeps FP64 masses.  The two handles take the same
mesh but for one point, whose mass is out of the pairs' range in one of them;
forces are the same bits, so accelerations differ by the products alone."""
import numpy as np
import pytest

from axisem_gb300 import _abi
from axisem_gb300.mesh import coupled_mesh, gvec_to_elemental, random_gvec
from axisem_gb300.solver import Solver

pytestmark = pytest.mark.gpu

SMALL, PATCHED = (23, 17, 5), (367, 359, 5)   # scattered; patched


def _masses(m, kind, scale, seed=3):
    """FP64 inverse masses of a mesh: `scale` times its FP32 ones with a
    remainder below their last bit.  kind: "pair"; "fp64" (one point out of the pairs' range, so that
    all products are FP64); "fp32" (the remainder dropped)."""
    rng = np.random.default_rng(seed)

    def dp(single, ig, ng):
        g = np.empty(ng)
        g[ig - 1] = np.asarray(single, np.float64).reshape(-1, order="F")
        g *= scale * (1.0 + rng.uniform(-1.0, 1.0, ng) * 2.0 ** -25)
        if kind == "fp32":
            g = g.astype(np.float32).astype(np.float64)
        g[ig[25 * 3 + 12] - 1] = 1e-40 if kind == "fp64" else 0.0
        return g

    s, f = dp(m.inv_mass_rho, m.igloc_solid, m.nglob_solid), dp(m.inv_mass_fluid, m.igloc_fluid, m.nglob_fluid)
    m.inv_mass_rho_dp = gvec_to_elemental(m, s)
    m.inv_mass_fluid_dp = gvec_to_elemental(m, f, fluid=True)


def _step(size, pole, kind, u, scale=1.0):
    """Accelerations of the first compensated step from the displacement u (but
    those of the point the handles hold apart)."""
    m = coupled_mesh(*size, pole, niter=4, terms="pole")
    m.magnitude = 1e37
    _masses(m, kind, scale)
    with Solver(m) as s:
        s.set_compensated(True)
        s.upload_disp(u)
        s.run(1, 1)
        a, b = s.get_state(_abi.FIELD_ACC0), s.get_state(_abi.FIELD_DDCHI0)
    a[2, 2, 3] = 0.0
    b[2, 2, 3] = 0.0
    return np.concatenate([a.ravel(order="K"), b.ravel(order="K")])


def _ulps(a, b):
    ia, ib = (x.view(np.int32).astype(np.int64) for x in (a, b))
    order = lambda i: np.where(i < 0, -(i & 0x7FFFFFFF), i)
    return np.abs(order(ia) - order(ib))


@pytest.mark.parametrize("size", [SMALL, PATCHED])
@pytest.mark.parametrize("pole", [0, 1, 2])
def test_mass_pair_products(gpu_lib, pole, size):
    """A pair's product is the FP64 product rounded once, but for values within
    2^-20 of an ulp from a tie: at most one unit in the last place anywhere, and
    equal at all but about 2^-19 of the values (1e-4 allowed: a coupled point
    takes several fluid accelerations).  FP32 masses, off by up to half a last
    bit, are not within that."""
    m = coupled_mesh(*size, pole, niter=4, terms="pole")
    u = random_gvec(m, seed=9)
    want = _step(size, pole, "fp64", u)
    got, single = _step(size, pole, "pair", u), _step(size, pole, "fp32", u)
    assert np.count_nonzero(want) > 0.3 * want.size
    assert _ulps(got, want).max() <= 1
    assert np.count_nonzero(got != want) <= 1e-4 * want.size
    assert np.count_nonzero(single != want) > 0.1 * np.count_nonzero(want)


@pytest.mark.parametrize("size", [SMALL, PATCHED])
def test_mass_pair_products_of_small_forces(gpu_lib, size):
    """Accelerations near 2^-110, whose rounding error FP32 does not hold."""
    m = coupled_mesh(*size, 2, niter=4, terms="pole")
    u = random_gvec(m, seed=9, sigma=1.0)
    scale = 1e-14   # (inverse masses of 1e-18 and more: displacements and forces stay far above 2^-126)
    a = np.abs(_step(size, 2, "fp64", u, scale))
    u = (u * (2.0 ** -110 / np.median(a[a > 0]))).astype(np.float32)
    want, got = _step(size, 2, "fp64", u, scale), _step(size, 2, "pair", u, scale)
    # (an acceleration below 2^-126 is zero to every later FP32 operation)
    normal = np.abs(want) >= 2.0 ** -126
    assert np.count_nonzero(normal) > 0.3 * want.size
    assert _ulps(got[normal], want[normal]).max() <= 1
    assert np.count_nonzero(got[normal] != want[normal]) <= 1e-4 * want.size


@pytest.mark.parametrize("size", [SMALL, PATCHED])
def test_mass_pair_products_of_infinite_forces(gpu_lib, size):
    """Where a force overflows, the acceleration is infinite, as with FP64
    masses.  (The displaced point is an element's corner, which the blow-up
    guard does not read.)"""
    m = coupled_mesh(*size, 2, niter=4, terms="pole")
    p = m.igloc_solid[25 * 40] - 1
    u = np.zeros((m.nglob_solid, 3), np.float32, order="F")
    u[p, 0] = 1.0
    with Solver(m) as s:
        f = np.abs(s.stiffness_assembled(u)).max()
    u[p, 0] = np.float32(1.5 * 3.4e38 / float(f))
    assert np.isfinite(u).all()
    want, got = _step(size, 2, "fp64", u), _step(size, 2, "pair", u)
    assert np.isinf(want).any()
    assert np.array_equal(np.isinf(got), np.isinf(want)) and np.array_equal(np.isnan(got), np.isnan(want))
