"""The work this framework is used for, as measurable cases.

A case is a dict of plain values:

  kind    "force": one stiffness + assembly through the C-ABI with pinned host
          buffers (axg_stiffness_assembled); "loop": `steps` time steps of one
          solve (axg_run) and its seismograms; "batch": the same for several
          solves advanced together (axg_batch_*).
  mesh    "grid": a structured solid layer of ni x nj elements over a fluid
          layer of ni x nf, the I = 0 column on the axis; "prem": the
          whole-Earth PREM mesh of `period` seconds.
  pole    0 monopole, 1 dipole, 2 quadrupole.
  mode    "plain", "comp" (compensated time integration), "cg4" (attenuation
          with 5 standard linear solids), "symplec4" (4-stage symplectic).
  dump    steps between displ_only wavefield snapshots (0: none), of the
          points dlo..dhi of each element in both directions.

Meshes stay resident, as a server keeps them: prepare() makes a new solve on
the mesh (axg_create_sharing) with a source, receivers and an initial
displacement of its own, drawn from the seed.  A pass advances that solve by
`steps` further steps, so its wavefield fills the mesh as in a long run.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from axisem_gb300 import _abi, sphere
from axisem_gb300.mesh import Mesh, add_attenuation, add_pointwise, gauss_at, gauss_stf, structured_igloc
from axisem_gb300.solver import Batch, Solver
from axisem_gb300.spectral import Spectral

N_TERMS = (15, 24, 26)   # metric arrays a solid element reads, per pole
N_AXIAL = (3, 9, 6)      # axial vectors
N_COMP = (2, 3, 3)       # displacement components
N_SLS = 5
# multiplications and additions per GLL point and step: the 5-term contractions
# of both stages and the pointwise products
FLOPS = (8 * 10 + 50, 12 * 10 + 110, 12 * 10 + 130)
FLOPS_FLUID = 4 * 10 + 8
COURANT = 0.3            # white noise holds every mode of the mesh: half the usual number keeps them all stable
SOURCE = {0: "explosion", 1: "mtr", 2: "mtp"}


# ------------------------------------------------------------------ the cases

def _loop(name, **kw):
    c = {"name": name, "kind": "loop", "mode": "plain", "dump": 0, "dlo": 0, "dhi": 4, "nrec": 200, "seis": 4}
    c.update(kw)
    return c


def listed():
    return [
        # one stiffness evaluation of a small mesh by a host program: launch and copy latency
        {"name": "force_di_small", "kind": "force", "mesh": "grid", "pole": 1, "ni": 37, "nj": 29, "nf": 0},
        # the headline stiffness + assembly, 2^20 quadrupole elements, end to end
        {"name": "force_quad_1m", "kind": "force", "mesh": "grid", "pole": 2, "ni": 1024, "nj": 1024, "nf": 0},
        # a toy run (tutorials, regression tests): a few dozen elements, absorbing boundaries
        _loop("loop_tiny", mesh="grid", pole=1, ni=9, nj=5, nf=3, absorbing=True, steps=250, nrec=6),
        # the default low-frequency whole-Earth run: PREM at 50 s, explosion
        _loop("loop_prem50_mono", mesh="prem", period=50, pole=0, steps=400),
        # the server's mode: compensated, PREM at 25 s
        _loop("loop_prem25_quad_comp", mesh="prem", period=25, pole=2, mode="comp", steps=200),
        # the anelastic production run: PREM at 10 s, dipole, 5 standard linear solids
        _loop("loop_prem10_di_cg4", mesh="prem", period=10, pole=1, mode="cg4", steps=72),
        # kernel wavefields: displacement snapshots of every point every 8 steps
        _loop("loop_prem25_di_dump", mesh="prem", period=25, pole=1, steps=128, dump=8),
        # a symplectic run on a mid-size mesh with ragged sides
        _loop("loop_grid_quad_symp", mesh="grid", pole=2, ni=211, nj=131, nf=45, mode="symplec4", steps=24),
        # a large anelastic mesh with ragged sides
        _loop("loop_grid_di_cg4", mesh="grid", pole=1, ni=701, nj=397, nf=131, mode="cg4", steps=36),
        # a large monopole run (the fewest bytes per element)
        _loop("loop_grid_mono", mesh="grid", pole=0, ni=1283, nj=611, nf=203, steps=40),
        # the largest: a mesh of about 2 s period, with sparse snapshots
        _loop("loop_grid_quad_1m", mesh="grid", pole=2, ni=1024, nj=768, nf=256, steps=32,
              dump=32, dlo=2, dhi=2),
        # served together: six compensated solves of both coarse PREM meshes and all poles
        {"name": "batch_prem_6", "kind": "batch", "mesh": "prem", "period": 50, "period2": 25, "solves": 6,
         "mode": "comp", "dump": 0, "dlo": 0, "dhi": 4, "steps": 96, "nrec": 60, "seis": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind, then sizes spread over the logarithm of the range."""
    u = rng.random()
    pole = rng.randrange(3)
    if u < 0.15:
        n = _log(rng, 200, 700000)
        ni = max(5, int(math.sqrt(n) * rng.uniform(0.6, 1.6)))
        return {"kind": "force", "mesh": "grid", "pole": pole, "ni": ni, "nj": max(3, n // ni), "nf": 0}
    mode = rng.choice(("plain", "plain", "comp", "cg4", "symplec4"))
    c = _loop("", nrec=rng.choice((1, 20, 60, 200)), seis=rng.randint(1, 7), pole=pole, mode=mode)
    del c["name"]
    if u < 0.35:
        c.update(mesh="prem", period=rng.choice((50, 25)), steps=rng.randint(40, 160))
    elif u < 0.5:
        return {"kind": "batch", "mesh": "prem", "period": 50, "period2": rng.choice((50, 25)),
                "solves": rng.randint(2, 7), "mode": rng.choice(("plain", "comp")), "dump": 0, "dlo": 0, "dhi": 4,
                "steps": rng.randint(24, 96), "nrec": rng.choice((20, 60)), "seis": rng.randint(1, 7)}
    else:
        n = _log(rng, 60, 400000)
        ni = max(5, int(math.sqrt(n) * rng.uniform(0.6, 1.6)))
        rows = max(6, n // ni)
        nf = max(2, int(rows * rng.uniform(0.1, 0.35)))
        c.update(mesh="grid", ni=ni, nj=rows - nf, nf=nf, absorbing=mode == "plain" and rng.random() < 0.3)
        c["steps"] = max(8, min(200, int(4e6 / n))) + rng.randint(0, 7)
    if mode == "symplec4":
        c["steps"] = max(6, c["steps"] // 4)
    if mode == "plain" and rng.random() < 0.3:
        lo = rng.randint(0, 2)
        c.update(dump=rng.randint(4, 12), dlo=lo, dhi=rng.randint(lo, 4))
    return c


# ------------------------------------------------------------------ meshes

_MESHES: dict = {}
_SKELETONS: dict = {}
_HOLDERS: dict = {}


def _f(a):
    return np.asfortranarray(a, dtype=np.float32)


def _grid(c):
    """The structured coupled mesh: metric terms, masses and boundary terms of
    physical scale (moduli near 1e11 Pa, densities 2500..13000 kg/m^3) whose
    quadratic form is positive, so that long runs stay bounded."""
    pole, ni, nj, nf = c["pole"], c["ni"], c["nj"], c["nf"]
    rng = np.random.default_rng([pole, ni, nj, nf])
    spec = Spectral()
    nel = ni * nj
    igloc, nglob = structured_igloc(ni, nj)
    wt2 = np.outer(spec.wt, spec.wt).astype(np.float32)

    def rnd(lo, hi, n):
        a = rng.random((n, 5, 5), dtype=np.float32)
        a *= np.float32(hi - lo)
        a += np.float32(lo)
        return a

    def to_f(a):   # (n, jpol, ipol), ipol fastest -> Fortran (ipol, jpol, n) without a copy
        return a.transpose(2, 1, 0)

    def points(values, ig):   # a per-point array as its element copies
        return np.asfortranarray(values.astype(np.float32)[ig - 1].reshape(-1, 5, 5).transpose(2, 1, 0))

    modulus = rnd(1e11, 3e11, nel) * wt2
    diagonal = {"M21s", "M41s", "M21z", "M41z", "M2phi", "M4phi", "M43s", "M33s", "M_w1", "M_w4", "M_w5"}
    if pole == 1:   # the dipole's M_w1 and M_w3 weigh u2 and u3
        diagonal = (diagonal | {"M_w3"}) - {"M33s", "M43s"}
    m_solid = {}
    for name in _abi.SOLID_TERMS_USED[pole]:
        m_solid[name] = to_f(modulus * (rnd(1.0, 2.0, nel) if name in diagonal else rnd(-0.07, 0.07, nel)))
    m0 = {}
    for name in _abi.AXIAL_TERMS_USED[pole]:
        on = name in {0: ("M0_w1",), 1: ("M0_w1",), 2: ("M0_w1", "M0_w4", "M0_w6")}[pole]
        r = rng.random((nel, 5), dtype=np.float32)
        m0[name] = (1e9 * (r + 0.5 if on else 0.02 * (r - 0.5))).astype(np.float32).T
    # assembled masses: a point's mass is that of the elements around it
    rho = rng.uniform(2500.0, 13000.0, nglob)
    inv = points(1.0 / (rho * float(wt2.mean())), igloc)
    m = Mesh(src_type=pole, nel_solid=nel, nglob_solid=nglob, igloc_solid=igloc,
             ax_el_solid=(np.arange(nj) * ni + 1).astype(np.int32), spec=spec, m_solid=m_solid, m0_solid=m0,
             inv_mass_rho=inv)
    if nf > 0:
        nelf = ni * nf
        igf, ngf = structured_igloc(ni, nf)
        m.nel_fluid, m.nglob_fluid, m.igloc_fluid = nelf, ngf, igf
        m.ax_el_fluid = (np.arange(nf) * ni + 1).astype(np.int32)
        for name in _abi.FLUID_TERMS[: 3 if pole == 0 else 4]:
            lo, hi = {"M1chi_fl": (-0.4, 0.4), "M2chi_fl": (1.0, 2.0), "M4chi_fl": (1.0, 2.0), "M_w_fl": (0.0, 0.5)}[name]
            m.m_fluid[name] = to_f(rnd(lo * 1e-2, hi * 1e-2, nelf) * wt2)
        m.m0_w_fl = (1e-4 * rng.random((nelf, 5), dtype=np.float32)).T
        m.inv_mass_fluid = points(rng.uniform(0.5e10, 2e10, ngf), igf)
        m.bdry_fluid_el = ((nf - 1) * ni + np.arange(ni) + 1).astype(np.int32)
        m.bdry_solid_el = (np.arange(ni) + 1).astype(np.int32)
        m.bdry_jpol_fluid = np.full(ni, 4, dtype=np.int32)
        m.bdry_jpol_solid = np.zeros(ni, dtype=np.int32)
        m.bdry_matr = _f(0.3 * rng.uniform(-1.0, 1.0, size=(5, ni, 2)))
    if c.get("absorbing"):
        m.solid_absorbing_gamma = points(10.0 * rng.random(nglob), igloc)
        if nf > 0:
            m.fluid_absorbing_gamma = points(10.0 * rng.random(ngf), igf)
    m.deltat = 1e-5
    if c.get("mode") == "cg4":
        add_attenuation(m, n_sls=N_SLS, seed=ni)
        for name in ("delta_mu_cg4", "delta_kappa_cg4"):   # small against the moduli: long runs stay bounded
            m.anel[name] = _f(m.anel[name] * 2e-3)
    if c.get("dump"):
        add_pointwise(m, seed=nj)
    return m


def _mesh(c):
    """The resident mesh of a case (and, on first use, its place in the cache)."""
    key = (c["mesh"], c["pole"], c.get("period"), c.get("ni"), c.get("nj"), c.get("nf"), c.get("mode") == "cg4",
           bool(c.get("dump")), bool(c.get("absorbing")))
    if key not in _MESHES:
        if c["mesh"] == "grid":
            _MESHES[key] = _grid(c)
        else:
            p = c["period"]
            if p not in _SKELETONS:
                _SKELETONS[p] = sphere.build_skeleton(float(p))
            _MESHES[key] = sphere.build_mesh(
                float(p), sphere.SphereSolve(pole=c["pole"], source=SOURCE[c["pole"]], seconds=float(p),
                                             receivers_deg=np.array([90.0]), courant=COURANT),
                skeleton=_SKELETONS[p], pointwise=bool(c.get("dump")),
                attenuation=sphere.Attenuation(n_sls=N_SLS) if c.get("mode") == "cg4" else None)
    return key, _MESHES[key]


def _axis_points(igloc, axial):
    """Global points (0-based) at ipol = 0 of the axial elements."""
    if axial is None or len(axial) == 0:
        return np.zeros(0, dtype=np.int64)
    return np.unique(igloc.reshape(-1, 5, 5)[np.asarray(axial) - 1, :, 0]) - 1


MASKED = ((0,), (1, 2), (0, 1, 2))   # components the axis mask zeroes, per pole


def _solve(c, seed):
    """The mesh with the solve's own source and receivers, and its initial
    displacement (nglob, 3): white noise, zero where the axis mask zeroes it."""
    key, base = _mesh(c)
    rng = np.random.default_rng([seed, c["pole"], 77])
    pole, steps = c["pole"], c.get("steps", 0)
    u = np.empty((3, base.nglob_solid), dtype=np.float32)
    if c["mesh"] == "prem":
        nrec = c["nrec"]
        solve = sphere.SphereSolve(pole=pole, source=SOURCE[pole], depth_km=float(rng.uniform(5.0, 600.0)),
                                   seconds=(steps - 0.5) * base.deltat,
                                   receivers_deg=np.sort(rng.uniform(0.0, 180.0, nrec)), seis_it=c["seis"])
        m = sphere.with_solve(base, solve, _SKELETONS[c["period"]])
        scale = 1e-3
    else:
        m = Mesh(**{k: getattr(base, k) for k in base.__dataclass_fields__})
        if steps:
            ni, nj = c["ni"], c["nj"]
            col, row = int(rng.integers(1, ni)), int(rng.integers(1, nj))
            val = rng.uniform(-1.0, 1.0, 3) * 1e3
            if pole == 0:
                val[1] = 0.0
            m.ielsrc = np.zeros(8, dtype=np.int32)
            m.source_term_el = np.zeros((5, 5, 8, 3), dtype=np.float32, order="F")
            corners = ((row - 1, col - 1, 4, 4), (row - 1, col, 0, 4), (row, col - 1, 4, 0), (row, col, 0, 0))
            for k, (r, q, ip, jp) in enumerate(corners):   # the four elements that hold the point
                m.ielsrc[k] = r * ni + q + 1
                m.source_term_el[ip, jp, k, :] = val
            m.nelsrc = 4
            m.stf = gauss_stf(steps, m.deltat, 20 * m.deltat)
            m.seis_it = c["seis"]
            n = c["nrec"]   # receivers anywhere in the solid
            m.recfile_el = np.asfortranarray(np.stack(
                [rng.integers(1, ni * nj + 1, n), rng.integers(0, 5, n), rng.integers(0, 5, n)], axis=1).astype(np.int32))
        scale = 1e-6
    for k in range(3):
        rng.standard_normal(out=u[k], dtype=np.float32)
    u *= np.float32(scale)
    if pole == 0:
        u[1] = 0.0
    if c["kind"] != "force":
        axis = _axis_points(m.igloc_solid, m.ax_el_solid)
        for k in MASKED[pole]:
            u[k, axis] = 0.0
    return key, m, u


def _members(c, seed):
    """The single solves a case stands for, and the seed of each."""
    if c["kind"] != "batch":
        return [(c, seed)]
    return [({**c, "kind": "loop", "period": c["period"] if k % 2 == 0 else c["period2"], "pole": k % 3},
             [seed, k]) for k in range(c["solves"])]


def _flat_seed(s):
    return s if isinstance(s, int) else int(s[0]) * 1000003 + int(s[1])


# ------------------------------------------------------------------ the path

def _ptr(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_float))


def _solver(c, seed):
    key, m, u = _solve(c, _flat_seed(seed))
    if key not in _HOLDERS:   # the mesh's arrays on the GPU, once
        _HOLDERS[key] = Solver(m)
    s = Solver(m, share_with=_HOLDERS[key])
    if c.get("mode") == "comp":
        s.set_compensated(True)
    if c.get("mode") == "symplec4":
        cd, _ = _pefrl(m.deltat)
        t = np.arange(m.niter)[:, None] * m.deltat + np.cumsum(cd[:-1])[None, :]
        s.set_time_scheme(_abi.SCHEME_SYMPLEC4, _stf_stages(c, m, t))
    st = {"s": s, "m": m}
    if c.get("dump"):
        lo, hi = c["dlo"], c["dhi"]
        floats = (hi - lo + 1) ** 2 * (N_COMP[c["pole"]] * (m.nel_solid + m.nel_fluid))
        cap = m.niter // c["dump"]
        out = torch.zeros((cap, floats), dtype=torch.float32, pin_memory=torch.cuda.is_available())
        s.set_wavefield_dump(_abi.DUMP_DISPL_ONLY, c["dump"], capacity=cap, ibeg=lo, iend=hi, jbeg=lo, jend=hi,
                             out=out.numpy())
        st["dump"] = out
    return st, u


def prepare(case, seed):
    if case["kind"] == "force":
        st, u = _solver(case, seed)
        st["u"] = torch.from_numpy(u).pin_memory()
        st["f"] = torch.empty_like(st["u"]).pin_memory()
        return st
    solves = []
    for c, s in _members(case, seed):
        st, u = _solver(c, s)
        st["s"].upload_disp(u.T)
        solves.append(st)
    state = {"solves": solves, "steps": case["steps"]}
    if case["kind"] == "batch":
        state["batch"] = Batch([st["s"] for st in solves])
    return state


def run(state):
    if "f" in state:
        s = state["s"]
        rc = s.lib.axg_stiffness_assembled(s.h, _ptr(state["u"]), _ptr(state["f"]))
        if rc:
            raise RuntimeError(s.lib.axg_last_error(s.h).decode())
        return state["f"]
    if "batch" in state:
        state["batch"].run([1] * len(state["solves"]), state["steps"])
    else:
        state["solves"][0]["s"].run(1, state["steps"])
    out = {}
    for k, st in enumerate(state["solves"]):
        out[f"seismograms{k}"] = st["s"].receivers()
        if "dump" in st:
            out[f"wavefield{k}"] = st["dump"]
    return out


def work(case):
    """Metric terms, numbering and boundary terms read once per step (per
    stage of a symplectic step), the state read and written once per point."""
    total = {"bytes": 0.0, "flops": 0.0}
    for c, _ in _members(case, 0):
        pole = c["pole"]
        if c["mesh"] == "grid":
            es, ef = c["ni"] * c["nj"], c["ni"] * c["nf"]
            gs, gf = (4 * c["ni"] + 1) * (4 * c["nj"] + 1), (4 * c["ni"] + 1) * (4 * c["nf"] + 1) if ef else 0
            ax, nb = c["nj"], c["ni"] if ef else 0
        else:
            es, ef = {50: (5664, 896), 25: (18944, 3200), 10: (99450, 17160)}[c["period"]]
            gs, gf, ax, nb = 16 * es, 16 * ef, int(math.sqrt(es)), int(2 * math.sqrt(ef))
        metric = es * (100 * N_TERMS[pole] + 100) + ax * 20 * N_AXIAL[pole]
        flops = es * 25 * FLOPS[pole] + ef * 25 * FLOPS_FLUID
        if c["kind"] == "force":
            total["bytes"] += metric + gs * 8 * N_COMP[pole]
            total["flops"] += flops
            continue
        state = 24 + (16 if c["mode"] == "comp" else 0)
        per = metric + gs * (state * N_COMP[pole] + 4) + ef * (100 * (3 if pole == 0 else 4) + 100)
        per += gf * (state + 4) + nb * 56
        if c["mode"] == "cg4":
            ne = 4 if pole == 0 else 6
            per += es * (4 * ne * N_SLS * 8 + 4 * (1 + ne) * 8 + 200)
        n = c["steps"] * (4 if c["mode"] == "symplec4" else 1)
        total["bytes"] += n * per
        total["flops"] += n * flops
        if c["dump"]:
            pts = (c["dhi"] - c["dlo"] + 1) ** 2
            total["bytes"] += (c["steps"] // c["dump"]) * pts * N_COMP[pole] * (es + ef) * 4
    return total


# ------------------------------------------------------------------ the same in 64 bits

def _pefrl(dt):
    """Drifts and kicks of the 4-stage symplectic scheme (Omelyan, Mryglod and
    Folk, 2002); its constants are single-precision ones."""
    z, i, k = (float(np.float32(x)) for x in (0.1786178958448091, -0.2123418310626054, -0.06626458266981849))
    return np.array([z, k, 1 - 2 * (z + k), k, z]) * dt, np.array([0.5 - i, i, i, 0.5 - i]) * dt


def _stf_stages(c, m, t):
    """The source time function at the stage times t (steps, stages)."""
    if c["mesh"] == "grid":
        return gauss_at(t, 20 * m.deltat)
    at = np.arange(1, m.niter + 1) * m.deltat
    return np.interp(t, at, m.stf).astype(np.float32)


class _Exact:
    """One solve in FP64 torch operations: the element-local formulas of the
    stiffness, anelastic and fluid terms on (element, j, i) arrays, assembled
    by index_add."""

    def __init__(self, c, m, u):
        self.c, self.m, self.pole = c, m, c["pole"]
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.ig = self.index(m.igloc_solid)
        self.ax = self.index(m.ax_el_solid)
        self.M = {k: self.elem(m.m_solid[k]) for k in _abi.SOLID_TERMS_USED[self.pole]}
        self.M0 = {k: self.real(np.asarray(m.m0_solid[k]).T)[self.ax] for k in _abi.AXIAL_TERMS_USED[self.pole]}
        sp = m.spec
        self.G1, self.G2, self.G0 = (self.real(sp.f32(k)) for k in ("G1", "G2", "G0"))
        self.u = self.real(u)

    def real(self, a):
        return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(self.dev)

    def index(self, a):
        n = [] if a is None else a
        return torch.from_numpy(np.asarray(n, dtype=np.int64) - 1).to(self.dev)

    def elem(self, a):   # Fortran (i, j, n) -> (n, j, i)
        return self.real(np.asarray(a).transpose(2, 1, 0))

    # d/dxi and d/deta of an element-local field, and the transposed second stage
    def dxi(self, f, ax=None):
        x = f @ self.G2
        ax = self.ax if ax is None else ax
        x[ax] = f[ax] @ self.G1
        return x

    def deta(self, f):
        return self.G2.T @ f

    def back(self, s1, s2, ax=None):
        x = s1 @ self.G2.T
        ax = self.ax if ax is None else ax
        x[ax] = s1[ax] @ self.G1.T
        return x + self.G2 @ s2

    def stiffness(self, u):
        """Element-local force components of the masked displacement u[c] (n, j, i)
        and the first-stage derivatives."""
        M, pole = self.M, self.pole
        x = [self.dxi(f) for f in u]
        e = [self.deta(f) for f in u]
        ax, g0 = self.ax, self.G0
        ua = [f[ax] for f in u]
        V = [f @ g0 for f in ua]                       # (axial, j)
        W = [f[:, :, 0] @ self.G2 for f in ua]         # d/deta on the axis
        w = {int(k[4:]): v for k, v in self.M0.items()}
        out = lambda v: v[:, :, None] * g0             # noqa: E731  outer product with G0 over i
        if pole == 0:
            us, _, uz = u
            X1, X2, X3, X4 = x[0], x[2], e[0], e[2]
            ls = M["M_4"] * X4 + M["M_2"] * X3 + M["M_1"] * X1 + M["M_3"] * X2 + us * M["M_w1"]
            s1s = M["M11s"] * X3 + M["M21s"] * X1 + M["M12s"] * X4 + M["M22s"] * X2 + M["M_1"] * us
            s2s = M["M11s"] * X1 + M["M41s"] * X3 + M["M32s"] * X2 + M["M42s"] * X4 + M["M_2"] * us
            s1z = M["M11z"] * X4 + M["M21z"] * X2 + M["M32s"] * X3 + M["M22s"] * X1 + M["M_3"] * us
            s2z = M["M11z"] * X2 + M["M41z"] * X4 + M["M12s"] * X1 + M["M42s"] * X3 + M["M_4"] * us
            f = [ls + self.back(s1s, s2s), torch.zeros_like(ls), self.back(s1z, s2z)]
            f[0][ax] += out(w[1] * V[0] + w[3] * W[2] + w[2] * V[2])
            f[2][ax] += out(w[2] * V[0])
            f[2][ax, :, 0] += (w[3] * V[0]) @ self.G2.T
        elif pole == 1:
            u1, u2, u3 = u
            X1, X2, X3, X4, X5, X6 = *x, *e
            X7, X8 = X1 + X2, X4 + X5
            l2 = (M["M_8"] * X6 + M["M_7"] * X3 + M["M_1"] * X1 + M["M_5"] * X2 + M["M_2"] * X4 + M["M_6"] * X5
                  + M["M_w1"] * u2 + M["M_w2"] * u3)
            l3 = M["M_4"] * (X4 - X5) + M["M_3"] * (X1 - X2) + M["M_w2"] * u2 + M["M_w3"] * u3
            c = M["M13s"] * X6 + M["M32s"] * X3
            s1p = c + M["M_3"] * u3 + M["M11s"] * X4 + M["M21s"] * X1 + M["M12s"] * X5 + M["M22s"] * X2 + M["M_1"] * u2
            s1m = c - M["M_3"] * u3 + M["M11s"] * X5 + M["M21s"] * X2 + M["M12s"] * X4 + M["M22s"] * X1 + M["M_5"] * u2
            c = M["M33s"] * X3 + M["M43s"] * X6
            s2p = c + M["M_4"] * u3 + M["M11s"] * X1 + M["M41s"] * X4 + M["M12s"] * X2 + M["M42s"] * X5 + M["M_2"] * u2
            s2m = c - M["M_4"] * u3 + M["M11s"] * X2 + M["M41s"] * X5 + M["M12s"] * X1 + M["M42s"] * X4 + M["M_6"] * u2
            s1z = M["M33s"] * X8 + M["M32s"] * X7 + M["M11z"] * X6 + M["M21z"] * X3 + M["M_7"] * u2
            s2z = M["M13s"] * X7 + M["M43s"] * X8 + M["M11z"] * X3 + M["M41z"] * X6 + M["M_8"] * u2
            f = [self.back(s1p, s2p), self.back(s1m, s2m) + l2, self.back(s1z, s2z) + l3]
            f[0][ax] += out(w[1] * V[1] + w[3] * V[2])
            f[0][ax, :, 0] += ((w[2] + w[6]) * V[1] + (w[4] + w[8]) * V[2]) @ self.G2.T
            f[1][ax] += out(w[1] * V[0] + (w[2] + w[6]) * W[0] + w[9] * V[1] + w[10] * V[2])
            f[2][ax] += out(w[3] * V[0] + (w[4] + w[8]) * W[0] + w[7] * V[2] + w[10] * V[1])
        else:
            us, up, uz = u
            X1, X2, X3, X4, X5, X6 = *x, *e
            a = M["M_2"] * X4 + M["M_1"] * X1 + M["M_4"] * X6 + M["M_3"] * X3
            b = M["M_6"] * X5 + M["M_5"] * X2
            ls = a + 2 * b + M["M_w1"] * us + M["M_w2"] * up + 2 * M["M_w3"] * uz
            lp = -2 * a - b + M["M_w2"] * us + M["M_w4"] * up - M["M_w3"] * uz
            lz = 2 * (M["M_8"] * X5 + M["M_7"] * X2) + M["M_w3"] * (2 * us - up) + M["M_w5"] * uz
            d, g = us - 2 * up, 2 * us - up
            s1s = M["M11s"] * X4 + M["M21s"] * X1 + M["M12s"] * X6 + M["M22s"] * X3 + M["M_1"] * d
            s2s = M["M11s"] * X1 + M["M41s"] * X4 + M["M32s"] * X3 + M["M42s"] * X6 + M["M_2"] * d
            s1z = M["M11z"] * X6 + M["M21z"] * X3 + M["M32s"] * X4 + M["M22s"] * X1 + M["M_3"] * d
            s2z = M["M11z"] * X3 + M["M41z"] * X6 + M["M12s"] * X1 + M["M42s"] * X4 + M["M_4"] * d
            s1p = M["M1phi"] * X5 + M["M2phi"] * X2 + M["M_5"] * g + 2 * M["M_7"] * uz
            s2p = M["M1phi"] * X2 + M["M4phi"] * X5 + M["M_6"] * g + 2 * M["M_8"] * uz
            f = [ls + self.back(s1s, s2s), lp + self.back(s1p, s2p), lz + self.back(s1z, s2z)]
            f[0][ax] += out(w[1] * V[0] + w[2] * V[1] + w[3] * V[2])
            f[1][ax] += out(w[2] * V[0] + w[4] * V[1] + w[5] * V[2])
            f[2][ax] += out(w[3] * V[0] + w[5] * V[1] + w[6] * V[2])
        return f, x, e

    def local(self, u):
        """Element-local copies of u (3, nglob), axis-masked."""
        n = self.m.nel_solid
        v = [u[k][self.ig].reshape(n, 5, 5) for k in range(3)]
        for k in MASKED[self.pole]:
            v[k][self.ax, :, 0] = 0.0
        return v

    def assemble(self, f, ig, ng):
        return torch.zeros(ng, dtype=torch.float64, device=self.dev).index_add_(0, ig, f.reshape(-1))

    def force(self, u, anel=False):
        """pdistsum(mask(stiffness(mask(u)))) on the global points (3, nglob)."""
        v = self.local(u)
        f, x, e = self.stiffness(v)
        if anel:
            f = self.anelastic(f, v, x, e)
        for k in MASKED[self.pole]:
            f[k][self.ax, :, 0] = 0.0
        return torch.stack([self.assemble(q, self.ig, self.m.nglob_solid) for q in f])

    # ---- time loop

    def start(self):
        m, pole = self.m, self.pole
        first = lambda a, ig, ng: self.real(self.points(a, ig, ng))   # noqa: E731
        dp = self.c["mode"] == "comp" and m.inv_mass_rho_dp is not None
        self.inv = first(m.inv_mass_rho_dp if dp else m.inv_mass_rho, m.igloc_solid, m.nglob_solid)
        self.axis = torch.from_numpy(_axis_points(m.igloc_solid, m.ax_el_solid)).to(self.dev)
        self.v, self.a = torch.zeros_like(self.u), torch.zeros_like(self.u)
        self.gam = self.gamf = None
        if m.solid_absorbing_gamma is not None:
            self.gam = first(m.solid_absorbing_gamma, m.igloc_solid, m.nglob_solid)
        src = m.source_term_el_dp if dp and m.source_term_el_dp is not None else m.source_term_el
        ig = m.igloc_solid.reshape(-1, 5, 5)
        self.src = torch.zeros_like(self.u)
        for k in range(m.nelsrc):
            g = ig[m.ielsrc[k] - 1].reshape(-1) - 1
            val = np.stack([np.asarray(src)[:, :, k, q].T.reshape(-1) for q in range(3)])
            nz = np.any(np.asarray(m.source_term_el)[:, :, k, :] != 0, axis=2).T.reshape(-1)
            self.src[:, torch.from_numpy(g[nz].astype(np.int64)).to(self.dev)] = self.real(val[:, nz])
        if pole == 0:
            self.src[1] = 0
        self.rec = torch.from_numpy(np.array([ig[e - 1, jp, ip] - 1 for e, ip, jp in m.recfile_el])).to(self.dev)
        if m.nel_fluid:
            self.igf = self.index(m.igloc_fluid)
            self.axf = self.index(m.ax_el_fluid)
            self.axisf = torch.from_numpy(_axis_points(m.igloc_fluid, m.ax_el_fluid)).to(self.dev)
            self.F = [self.elem(m.m_fluid[k]) for k in _abi.FLUID_TERMS[: 3 if pole == 0 else 4]]
            if pole:
                self.F0 = self.real(np.asarray(m.m0_w_fl).T)[self.axf]
            dpf = self.c["mode"] == "comp" and m.inv_mass_fluid_dp is not None
            self.invf = first(m.inv_mass_fluid_dp if dpf else m.inv_mass_fluid, m.igloc_fluid, m.nglob_fluid)
            if m.fluid_absorbing_gamma is not None:
                self.gamf = first(m.fluid_absorbing_gamma, m.igloc_fluid, m.nglob_fluid)
            z = torch.zeros(m.nglob_fluid, dtype=torch.float64, device=self.dev)
            self.chi, self.dchi, self.ddchi = z, z.clone(), z.clone()
            es, ef = m.bdry_solid_el - 1, m.bdry_fluid_el - 1
            igf = m.igloc_fluid.reshape(-1, 5, 5)
            to = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int64)).to(self.dev)   # noqa: E731
            self.bs = to(ig[es, m.bdry_jpol_solid] - 1)       # (boundary, i)
            self.bf = to(igf[ef, m.bdry_jpol_fluid] - 1)
            self.b1, self.b2 = (self.real(np.asarray(m.bdry_matr)[:, :, k].T) for k in (0, 1))
            axs = np.zeros(m.nel_solid, bool)
            axs[m.ax_el_solid - 1] = True
            axf = np.zeros(m.nel_fluid, bool)
            if m.ax_el_fluid is not None:
                axf[m.ax_el_fluid - 1] = True
            keep = np.ones((len(es), 5))
            keep[axs[es], 0] = 0.0
            self.keep_s = self.real(keep)                     # the solid copy is not on the axis
            keep = np.ones((len(es), 5))
            if pole:
                keep[axf[ef], 0] = 0.0
            self.keep_f = self.real(keep)
        if self.c["mode"] == "cg4":
            a = m.anel
            self.A = {k: self.real(np.asarray(v).T) for k, v in a.items() if k.endswith("_cg4")}
            jj, ii = [1, 3, 1, 3], [1, 1, 3, 3]               # cg points (i, j) = (1,1), (1,3), (3,1), (3,3)
            self.cgj, self.cgi = jj, ii
            self.invs = self.elem(a["inv_s_solid"])[:, jj, ii]
            rows = {}
            for q in np.unique(np.concatenate([a["Q_mu"], a["Q_kappa"]])):
                y = np.asarray(a["y_j"], np.float64) / float(q)
                if a.get("do_corr_lowq"):
                    dy, yp = 1.0 + 0.5 * y[0], np.zeros_like(y)
                    yp[0] = y[0] * dy
                    for k in range(1, len(y)):
                        dy = dy + (dy - 0.5) * y[k - 1] + 0.5 * y[k]
                        yp[k] = y[k] * dy
                    y = yp
                rows[float(q)] = y / y.sum()
            fac = lambda Q, ts: self.real(np.stack([rows[float(q)] for q in Q]) * np.asarray(ts)[None])   # noqa: E731
            self.mu_t, self.mu_m = fac(a["Q_mu"], a["ts_fac_t"]), fac(a["Q_mu"], a["ts_fac_tm1"])
            self.ka_t, self.ka_m = fac(a["Q_kappa"], a["ts_fac_t"]), fac(a["Q_kappa"], a["ts_fac_tm1"])
            self.ex = self.real(a["exp_w_j_deltat"])
            n = m.nel_solid
            z = lambda *s: torch.zeros(s, dtype=torch.float64, device=self.dev)   # noqa: E731
            self.R, self.tr, self.dev6 = z(n, len(a["y_j"]), 6, 4), z(n, 4), z(n, 6, 4)

    @staticmethod
    def points(a, ig, ng):
        """Per-point values of an element-local array: the first copy's."""
        out = np.zeros(ng, dtype=np.float64)
        out[ig[::-1] - 1] = np.asarray(a).reshape(-1, order="F")[::-1]
        return out

    def anelastic(self, f, u, x, e):
        """Minus the anelastic stiffness of the summed memory variables, then
        their update from the strain at the four cg points."""
        pole, A = self.pole, self.A
        r = self.R.sum(1)                                     # (n, 6, 4)
        vse, vsx, vze, vzx, y = (A[k] for k in ("V_s_eta_cg4", "V_s_xi_cg4", "V_z_eta_cg4", "V_z_xi_cg4", "Y_cg4"))
        r0, r1, r2, r3, r4, r5 = (r[:, k] for k in range(6))
        full = lambda s: self.spread(s)                       # noqa: E731
        sub = lambda s1, s2: self.back(full(s1), full(s2))    # noqa: E731
        z = sub(vze * r4 + vse * r2, vzx * r4 + vsx * r2)
        if pole == 0:
            f[0] = f[0] - sub(vze * r0 + vse * r4, vzx * r0 + vsx * r4) - full(y * r1)
            f[2] = f[2] - z
        elif pole == 1:
            f[0] = f[0] - sub(vze * (r0 - r5) + vse * (r4 - r3), vzx * (r0 - r5) + vsx * (r4 - r3))
            f[1] = f[1] - sub(vze * (r0 + r5) + vse * (r4 + r3), vzx * (r0 + r5) + vsx * (r4 + r3)) - full(2 * y * (r1 - r5))
            f[2] = f[2] - z + full(y * r3)
        else:
            f[0] = f[0] - sub(vze * r0 + vse * r4, vzx * r0 + vsx * r4) - full(y * (r1 - 2 * r5))
            f[1] = f[1] + sub(vze * r5 + vse * r3, vzx * r5 + vsx * r3) - full(y * (r5 - 2 * r1))
            f[2] = f[2] - z + full(2 * y * r3)
        at = lambda q: q[:, self.cgj, self.cgi]               # noqa: E731
        gs = lambda p, q: A["DzDeta_over_J_sol_cg4"] * p + A["DzDxi_over_J_sol_cg4"] * q   # noqa: E731
        gz = lambda p, q: A["DsDeta_over_J_sol_cg4"] * p + A["DsDxi_over_J_sol_cg4"] * q   # noqa: E731
        X, E, U, s = [at(q) for q in x], [at(q) for q in e], [at(q) for q in u], self.invs
        zero = torch.zeros_like(s)
        b = (X[0] + X[1], E[0] + E[1]) if pole == 1 else (X[0], E[0])
        g0, g2, g4 = gs(*b), gz(X[2], E[2]), gz(*b) + gs(X[2], E[2])
        if pole == 0:
            g1, g3, g5 = s * U[0], zero, zero
        elif pole == 1:
            g1 = 2 * s * U[1]
            d = (X[0] - X[1], E[0] - E[1])
            g3, g5 = -s * U[2] - gz(*d), -g1 - gs(*d)
        else:
            g1 = s * (U[0] - 2 * U[1])
            g3, g5 = -2 * s * U[2] - gz(X[1], E[1]), s * (U[1] - 2 * U[0]) - gs(X[1], E[1])
        tr = g0 + g1 + g2
        dm = A["delta_mu_cg4"]
        new = torch.stack([2 * dm * (g0 - tr / 3), 2 * dm * (g1 - tr / 3), 2 * dm * (g2 - tr / 3), dm * g3, dm * g4, dm * g5], 1)
        k = A["delta_kappa_cg4"] * tr
        up = self.mu_t[:, :, None, None] * new[:, None] + self.mu_m[:, :, None, None] * self.dev6[:, None]
        bulk = self.ka_t[:, :, None] * k[:, None] + self.ka_m[:, :, None] * self.tr[:, None]
        up[:, :, :3] += bulk[:, :, None]
        self.R = self.ex[None, :, None, None] * self.R + up
        self.tr, self.dev6 = k, new
        return f

    def spread(self, s):   # cg-point values (n, 4) as an element field, zero elsewhere
        o = torch.zeros((s.shape[0], 5, 5), dtype=torch.float64, device=self.dev)
        o[:, self.cgj, self.cgi] = s
        return o

    def fluid_force(self, chi, u):
        """Fluid stiffness of chi plus the coupling from the displacement u."""
        m, pole = self.m, self.pole
        n = m.nel_fluid
        q = chi[self.igf].reshape(n, 5, 5)
        if pole:
            q[self.axf, :, 0] = 0.0
        X1, X2 = self.dxi(q, self.axf), self.deta(q)
        F = self.F
        f = self.back(F[0] * X2 + F[1] * X1, F[0] * X1 + F[2] * X2, self.axf)
        if pole:
            f = f + F[3] * q
            f[self.axf] += (self.F0 * (q[self.axf] @ self.G0))[:, :, None] * self.G0
            f[self.axf, :, 0] = 0.0
        f = self.assemble(f, self.igf, m.nglob_fluid)
        us = u[0][self.bs] + u[1][self.bs] if pole == 1 else u[0][self.bs]
        b = -self.keep_f * (self.b1 * us + self.b2 * u[2][self.bs])
        return f.index_add_(0, self.bf.reshape(-1), b.reshape(-1))

    def solid_force(self, u, ddchi, stf, anel):
        f = self.force(u, anel)
        if self.m.nel_fluid:
            a = ddchi[self.bf]
            t = [self.b1 * a, self.b1 * a if self.pole == 1 else None, self.b2 * a]
            for k in range(3):
                if t[k] is not None:
                    q = t[k] * self.keep_s if k in MASKED[self.pole] else t[k]
                    f[k].index_add_(0, self.bs.reshape(-1), q.reshape(-1))
        return f - self.src * stf

    def masked(self, u):
        u = u.clone()
        for k in MASKED[self.pole]:
            u[k, self.axis] = 0.0
        return u

    def loop(self):
        """All steps; returns the seismograms and the snapshots."""
        m, c, pole = self.m, self.c, self.pole
        self.start()
        dt, ns = m.deltat, m.niter // m.seis_it + 1
        rec = np.zeros((ns, 3, m.num_rec))
        snaps = []
        sym = c["mode"] == "symplec4"
        if sym:
            cd, cv = _pefrl(dt)
            stf = _stf_stages(c, m, np.arange(m.niter)[:, None] * dt + np.cumsum(cd[:-1])[None, :])
        two = torch.ones((3, 1), dtype=torch.float64, device=self.dev)
        if pole == 1:
            two[2] = 2.0
        for it in range(1, m.niter + 1):
            if sym:
                for k in range(len(cv)):
                    u = self.u + cd[k] * self.v
                    if m.nel_fluid:
                        chi = self.chi + cd[k] * self.dchi
                        self.ddchi = -self.invf * self.fluid_force(chi, u)
                        self.dchi = self.dchi + cv[k] * self.ddchi
                        if pole:
                            chi[self.axisf] = 0.0
                        self.chi = chi
                    u = self.masked(u)
                    acc = -self.inv * self.solid_force(u, self.ddchi if m.nel_fluid else None, float(stf[it - 1, k]), False)
                    self.u, self.v = u, self.v + cv[k] * two * acc
                self.u = self.u + cd[-1] * self.v
                if m.nel_fluid:
                    self.chi = self.chi + cd[-1] * self.dchi
            else:
                u = self.u + dt * self.v + 0.5 * dt * dt * self.a
                if m.nel_fluid:
                    chi = self.chi + dt * self.dchi + 0.5 * dt * dt * self.ddchi
                    acc = -self.invf * self.fluid_force(chi, u)
                    if self.gamf is not None:
                        acc = acc - 2 * self.gamf * self.dchi - self.gamf ** 2 * chi
                    self.dchi = self.dchi + 0.5 * dt * (self.ddchi + acc)
                    self.ddchi = acc
                    if pole:
                        chi[self.axisf] = 0.0
                    self.chi = chi
                free, u = u, self.masked(u)
                acc = -self.inv * two * self.solid_force(u, self.ddchi if m.nel_fluid else None,
                                                         float(m.stf[it - 1]), c["mode"] == "cg4")
                if self.gam is not None:
                    acc = acc - 2 * self.gam * self.v - self.gam ** 2 * free
                self.v = self.v + 0.5 * dt * (self.a + acc)
                self.u, self.a = u, acc
            if it % m.seis_it == 0:
                w = self.u[:, self.rec].cpu().numpy()
                if pole == 0:
                    w[1] = 0.0
                if pole == 1:
                    w[0], w[1] = w[0] + w[1], w[0] - w[1]
                rec[it // m.seis_it] = w
            if c["dump"] and it % c["dump"] == 0:
                snaps.append(self.snapshot())
        return rec, np.stack(snaps) if snaps else None

    def snapshot(self):
        """dump_disp_global: (s, phi, z) of the solid, grad(chi) / rho of the fluid."""
        m, pole, lo, hi = self.m, self.pole, self.c["dlo"], self.c["dhi"] + 1
        cut = lambda q: q[:, lo:hi, lo:hi].reshape(-1).cpu().numpy()   # noqa: E731
        u = [self.u[k][self.ig].reshape(-1, 5, 5) for k in range(3)]
        u = {0: [u[0], u[2]], 1: [u[0] + u[1], u[0] - u[1], u[2]], 2: u}[pole]
        out = [cut(q) for q in u]
        if m.nel_fluid:
            P = {k: self.elem(v) for k, v in m.pointwise.items() if k.endswith(("_flu", "_fluid"))}
            q = self.chi[self.igf].reshape(-1, 5, 5)
            X, E, r = self.dxi(q, self.axf), self.deta(q), P["inv_rho_fluid"]
            s = r * (P["DzDeta_over_J_flu"] * X + P["DzDxi_over_J_flu"] * E)
            z = r * (P["DsDeta_over_J_flu"] * X + P["DsDxi_over_J_flu"] * E)
            out += [cut(q) for q in ([s, z] if pole == 0 else [s, torch.zeros_like(s), z])]
        return np.concatenate(out)


def exact(case, seed):
    if case["kind"] == "force":
        _, m, u = _solve(case, seed)
        return _Exact(case, m, u).force(torch.from_numpy(u.astype(np.float64)).to(
            "cuda" if torch.cuda.is_available() else "cpu")).cpu().numpy()
    out = {}
    for k, (c, s) in enumerate(_members(case, seed)):
        _, m, u = _solve(c, _flat_seed(s))
        rec, snaps = _Exact(c, m, u).loop()
        out[f"seismograms{k}"] = rec
        if c["dump"]:
            out[f"wavefield{k}"] = snaps
    return out
