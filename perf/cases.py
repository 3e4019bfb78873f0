"""The work a user of this framework has it do, as measurable cases.

Every case goes through the Python binding's public calls, as a host program
makes them: a solve advanced a few outer iterations and its fields read back
into pinned buffers (what a worker thread publishes), a batched polar, the
pressure CG primitive, the wall forces and streamlines of a field, and a
serving run of the engine. Grids are the C-grids of the tests and the
benchmark (192x48, 384x96, 768x192) and ragged ones between.

`listed()` names the cases, `draw(rng)` makes more of the same ranges,
`prepare(case, seed)` builds what a program holds before the call,
`run(state)` makes one pass, `work(case)` counts the bytes and operations a
pass cannot do without, and `exact(case, seed)` gives the pass's results from
plain numpy in 64 bits.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

_PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cfd-simulator_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import cfd_b200 as cb  # noqa: E402

EXTENTS = dict(upstream_chords=10.0, downstream_chords=15.0, vertical_chords=10.0)
COARSE = dict(surface=64, wake=33, normal=49)      # 192 x 48 cells
MEDIUM = dict(surface=128, wake=65, normal=97)     # 384 x 96
FINE = dict(surface=256, wake=129, normal=193)     # 768 x 192


# ---- the cases ------------------------------------------------------------------

def _solve(name=None, grid=MEDIUM, section="0012", first_layer=1e-5, alpha=4.0, reynolds=1e6, model="sst",
           precision="plain", scheme=0, iterations=2):
    case = dict(kind="solve", section=section, first_layer=first_layer, alpha=alpha, reynolds=reynolds,
                model=model, precision=precision, scheme=scheme, iterations=iterations, **grid)
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest ordinary solve: a laminar coarse grid, bound by the
        # latency of its dependent steps
        _solve("laminar_coarse", COARSE, first_layer=2e-3, alpha=0.0, reynolds=500.0, model="laminar"),
        # the medium turbulent solve most requests ask for
        _solve("sst_medium"),
        # the fine grid a published polar point is solved on
        _solve("sst_fine", FINE, "2412", 5e-6, 6.0, 3e6, iterations=1),
        # a user's own grid, no power of two anywhere, with the second-order scheme
        _solve("sst_ragged_second_order", dict(surface=77, wake=41, normal=62), "2412", 2e-5, 2.0, 1e6, scheme=1),
        # the mixed FP32/FP64 form, medium and fine
        _solve("mixed_medium", precision="mixed"),
        _solve("mixed_fine", FINE, "2412", 5e-6, 6.0, 3e6, precision="mixed"),
        # a polar: eight angles on the fine grid and three other grids beside
        # them, all advanced together
        dict(name="polar_batch", kind="batch", section="2412", points=8, alpha=-2.0, step=2.0, reynolds=3e6,
             first_layer=5e-6, trio=True, precision="plain", iterations=1, **FINE),
        # the pressure CG as a library call: the solver's own rule on a coarse
        # grid without allocation, and a tight solve on the fine grid
        dict(name="cg_coarse", kind="cg", cells_i=192, cells_j=48, wake=True, tolerance=0.01, cap=200, noalloc=True),
        dict(name="cg_fine", kind="cg", cells_i=768, cells_j=192, wake=True, tolerance=1e-8, cap=1000, noalloc=False),
        # post-processing of a field: wall forces (the smallest call) and the
        # streamlines a viewer draws
        dict(name="forces_fine", kind="forces", section="2412", first_layer=5e-6, alpha=6.0, reynolds=3e6, **FINE),
        dict(name="streamlines_medium", kind="streamlines", section="0012", first_layer=1e-5, alpha=4.0,
             reynolds=1e6, seeds=24, max_steps=1500, backwards=True, **MEDIUM),
        # serving: requests of several sections and angles through the engine,
        # grids built on its threads, mixed form
        dict(name="serve_coarse", kind="engine", requests=8, reynolds=1e6, first_layer=2e-3, iterations=32, **COARSE),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_grid(rng):
    return dict(surface=_log_int(rng, 24, 256), wake=_log_int(rng, 12, 128), normal=_log_int(rng, 14, 190))


def draw(rng):
    kind = rng.choices(["solve", "mixed", "batch", "cg", "forces", "streamlines"], [40, 16, 10, 20, 7, 7])[0]
    section = rng.choice(["0012", "2412", "0015", "4415"])
    alpha = round(rng.uniform(-4.0, 10.0), 2)
    reynolds = round(10 ** rng.uniform(5.3, 6.5))
    layer = 10 ** rng.uniform(-5.2, -3.5)
    if kind in ("solve", "mixed"):
        laminar, grid = rng.random() < 0.25, _draw_grid(rng)
        return _solve(None, grid, section, 2e-3 if laminar else layer, alpha,
                      round(rng.uniform(200, 800)) if laminar else reynolds, "laminar" if laminar else "sst",
                      "mixed" if kind == "mixed" else "plain", rng.choice([0, 0, 1]), 1 if _cells(grid) > 60000 else 2)
    if kind == "batch":
        return dict(kind="batch", section=section, points=rng.randint(2, 8), alpha=-2.0, step=1.5, reynolds=reynolds,
                    first_layer=layer, trio=rng.random() < 0.3, precision=rng.choice(["plain", "mixed"]),
                    iterations=1, **_draw_grid(rng))
    if kind == "cg":
        wake = rng.random() < 0.6
        ci = _log_int(rng, 20, 760)
        cj = _log_int(rng, 10, 190)
        ci += (ci & 1) if wake else 0  # a wake cut pairs its columns
        return dict(kind="cg", cells_i=ci, cells_j=cj, wake=wake, tolerance=rng.choice([0.01, 1e-4, 1e-8]),
                    cap=rng.choice([200, 1000]), noalloc=(ci + 1) * (cj + 1) <= 65536 and rng.random() < 0.5)
    case = dict(kind=kind, section=section, first_layer=layer, alpha=alpha, reynolds=reynolds, **_draw_grid(rng))
    if kind == "streamlines":
        case.update(seeds=rng.randint(5, 40), max_steps=_log_int(rng, 200, 1500), backwards=rng.random() < 0.7)
    return case


# ---- what a program has in hand -----------------------------------------------------

@functools.lru_cache(maxsize=8)
def _mesh(section, surface, wake, normal, first_layer):
    return cb.cgrid(section, surface_points=surface, wake_points=wake, normal_points=normal,
                    first_layer_height=first_layer, **EXTENTS)


def _case_mesh(case):
    return _mesh(case["section"], case["surface"], case["wake"], case["normal"], case["first_layer"])


def _settings(case):
    return cb.Settings.defaults(inflow_intensity=0.001, inflow_viscosity_ratio=10.0, scheme=case.get("scheme", 0),
                                precision=1 if case.get("precision") == "mixed" else 0)


def _start(mesh, alpha, reynolds, seed):
    """The freestream of a request (its angle and Reynolds number jittered)
    with a smooth disturbance of a percent: a start no two programs share."""
    rng = np.random.RandomState(seed % (1 << 31))
    alpha += rng.uniform(-0.5, 0.5)
    reynolds *= rng.uniform(0.9, 1.1)
    u, v, p, rho, mu = cb.uniform_field(mesh, 1.0, alpha, 1.0, reynolds)
    x, y = mesh.centroid[0::2], mesh.centroid[1::2]
    a, b, c = rng.uniform(0.5, 2.0, 3)
    ripple = 0.01 * np.sin(a * x + rng.uniform(0, 6)) * np.cos(b * y + rng.uniform(0, 6))
    return alpha, (u * (1.0 + ripple), v + 0.01 * np.cos(c * x) * np.exp(-0.1 * y * y), p, rho, mu)


MODELS = {"laminar": cb.MODEL_LAMINAR, "sst": cb.MODEL_SST}


def _solver(mesh, case, alpha, reynolds, seed, model):
    alpha, field = _start(mesh, alpha, reynolds, seed)
    s = cb.SimpleSolver.create(mesh, cb.freestream_conditions(mesh, 1.0, alpha), _settings(case))
    s.set_turbulence_model(MODELS[model])
    s.initialise(*field)
    return s, alpha


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def _batch_points(case):
    """(mesh, alpha, Reynolds number) of every solve of a batch."""
    points = [(_case_mesh(case), case["alpha"] + k * case["step"], case["reynolds"]) for k in range(case["points"])]
    if case["trio"]:
        for grid, layer in ((COARSE, 2e-3), (MEDIUM, 1e-5)):
            points.append((_mesh("0012", grid["surface"], grid["wake"], grid["normal"], layer), 4.0, 1e6))
    return points


def _cg_arrays(case, seed):
    """A pressure-correction system of a stretched grid: symmetric five-point
    couplings with strong anisotropy towards the wall, a pressure outlet on the
    outer rows, and mass imbalances as the source (numpy; reference order)."""
    ni, nj = case["cells_i"], case["cells_j"]
    rng = np.random.RandomState(seed % (1 << 31))
    stretch = 10.0 ** (2.0 * (1.0 - np.arange(nj + 1) / nj))
    north = stretch[:, None] * rng.uniform(0.5, 1.5, (nj + 1, ni))
    east = (1.0 / stretch[:nj])[:, None] * rng.uniform(0.5, 1.5, (nj, ni + 1))
    outlet = np.zeros((nj, ni))
    outlet[-1] = north[-1]
    outlet[:, 0] += east[:, 0]
    outlet[:, -1] += east[:, -1]
    north[0] = north[-1] = 0.0
    east[:, 0] = east[:, -1] = 0.0
    across = np.full(ni, -1, np.int32)
    if case["wake"]:
        cut = max(1, ni // 6)
        across[:cut] = ni - 1 - np.arange(cut)
        across[ni - cut:] = ni - 1 - np.arange(ni - cut, ni)
        pair = stretch[0] * rng.uniform(0.5, 1.5, cut)
        north[0, :cut] = pair
        north[0, ni - cut:] = pair[::-1]
    diag = north[:-1] + north[1:] + east[:, :-1] + east[:, 1:] + outlet
    upper = np.concatenate([-north.ravel(), -east.T.ravel()])
    return diag.ravel(), upper, rng.standard_normal(ni * nj), across


def _developed(mesh, alpha, seed):
    """A field with the features post-processing meets: a boundary layer along
    the section, a pressure peak at the nose, an eddy viscosity."""
    rng = np.random.RandomState(seed % (1 << 31))
    x, y = mesh.centroid[0::2], mesh.centroid[1::2]
    t = np.clip(x, 0.0, 1.0)
    d = np.hypot(x - t, y)
    layer = 1.0 - np.exp(-d / (0.02 + 0.03 * t + 0.01 * rng.random()))
    ux, uy = cb.freestream_velocity(1.0, alpha)
    near = np.exp(-2.0 * d)
    u = layer * (ux + 0.2 * near * np.sign(y) * math.sin(math.radians(alpha)) + 0.02 * np.sin(3 * x + rng.uniform(0, 6)))
    v = layer * (uy + 0.05 * near * (0.5 - t) * np.sign(y) + 0.02 * np.cos(2 * x + rng.uniform(0, 6)) * near)
    p = 0.5 * np.exp(-((x ** 2 + y ** 2) / 0.01)) - 0.3 * near * (y > 0) * (1 - t) + 0.01 * np.sin(5 * x) * near
    return u, v, p


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        mesh = _case_mesh(case)
        s, _ = _solver(mesh, case, case["alpha"], case["reynolds"], seed, case["model"])
        names = ["U", "V", "P"] + (["K", "OMEGA", "MUT"] if case["model"] == "sst" else [])
        return dict(kind=kind, solver=s, iterations=case["iterations"], out={n: _pinned(mesh.cells) for n in names})
    if kind == "batch":
        solvers = [_solver(mesh, case, alpha, re, seed + 7 * k, "sst")[0]
                   for k, (mesh, alpha, re) in enumerate(_batch_points(case))]
        out = [{n: _pinned(s.mesh.cells) for n in ("U", "V", "P")} for s in solvers]
        return dict(kind=kind, solvers=solvers, batch=cb.Batch(solvers), iterations=case["iterations"], out=out)
    if kind == "cg":
        diag, upper, source, across = _cg_arrays(case, seed)
        dev = {n: torch.tensor(a, device="cuda") for n, a in
               dict(diag=diag, upper=upper, source=source, across=across).items()}
        system = cb.CgSystem(case["cells_i"], case["cells_j"], dev["diag"].data_ptr(), dev["upper"].data_ptr(),
                             dev["source"].data_ptr(), dev["across"].data_ptr() if case["wake"] else None)
        x = torch.zeros(case["cells_i"] * case["cells_j"], dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return dict(kind=kind, call=cb.cg_solve_noalloc if case["noalloc"] else cb.cg_solve, system=system, dev=dev,
                    x=x, tolerance=case["tolerance"], cap=case["cap"])
    if kind in ("forces", "streamlines"):
        mesh = _case_mesh(case)
        s, alpha = _solver(mesh, case, case["alpha"], case["reynolds"], seed, "laminar")
        u, v, p = _developed(mesh, alpha, seed)
        s.load_state(u=u, v=v, p=p)
        state = dict(kind=kind, solver=s, alpha=alpha)
        if kind == "streamlines":
            state.update(seeds=_seeds(case, seed), max_steps=case["max_steps"], backwards=case["backwards"],
                         vertices=np.zeros((_vertices(case), 2)))
        return state
    rng = np.random.RandomState(seed % (1 << 31))
    requests = [cb.request(section, float(rng.uniform(-2, 8)), case["reynolds"] * rng.uniform(0.8, 1.2),
                           tolerance=1e-6, max_iterations=case["iterations"], surface_points=case["surface"],
                           wake_points=case["wake"], normal_points=case["normal"],
                           first_layer_height=case["first_layer"], **EXTENTS,
                           settings=cb.Settings.defaults(inflow_viscosity_ratio=10.0, precision=1))
                for section in [["0012", "2412", "0015", "4415"][k % 4] for k in range(case["requests"])]]
    return dict(kind=kind, requests=requests)


def _vertices(case):
    return case["seeds"] * (2 * case["max_steps"] + 1)


def _seeds(case, seed):
    rng = np.random.RandomState((seed + 1) % (1 << 31))
    n = case["seeds"]
    y = np.linspace(-1.2, 1.2, n) + rng.uniform(-0.02, 0.02, n)
    return np.stack([np.full(n, -1.5) + rng.uniform(-0.1, 0.1, n), y], 1)


# ---- one pass -----------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "solve":
        s = state["solver"]
        monitor = s.iterate(state["iterations"])
        for name, buffer in state["out"].items():
            s.read_into(name, buffer)
        return dict(state["out"], monitor=monitor.as_array())
    if kind == "batch":
        _, monitors = state["batch"].iterate(state["iterations"])
        for s, out in zip(state["solvers"], state["out"]):
            for name, buffer in out.items():
                s.read_into(name, buffer)
        return dict(fields=state["out"], monitors=np.stack([m.as_array() for m in monitors]))
    if kind == "cg":
        x = state["x"]
        x.zero_()
        report = state["call"](state["system"], x.data_ptr(), state["tolerance"], state["cap"])
        return dict(x=x, report=report[:3], converged=int(report[3]))
    if kind == "forces":
        f, cp, cf = state["solver"].forces(1.0, state["alpha"])
        return dict(coefficients=np.array([f.lift_coefficient, f.drag_coefficient, f.moment_coefficient,
                                           f.pressure_drag_coefficient, f.friction_drag_coefficient]),
                    cp=cp, cf=cf, stations=f.stations)
    if kind == "streamlines":
        lengths, points = state["solver"].streamlines(state["seeds"], max_steps=state["max_steps"],
                                                      trace_backwards=state["backwards"])
        vertices = state["vertices"]  # the viewer's vertex buffer, of fixed size
        vertices[:len(points)] = points
        vertices[len(points):] = 0.0
        return dict(lengths=lengths, vertices=vertices)
    engine = cb.Engine(chunk=16)
    results = engine.run(state["requests"])
    surfaces = [engine.surface(r.id) for r in results]
    engine.close()
    return dict(iterations=np.array([r.iterations for r in results]), status=np.array([r.status for r in results]),
                coefficients=np.array([[r.lift_coefficient, r.drag_coefficient, r.moment_coefficient]
                                       for r in results]), cp=np.concatenate(surfaces))


# ---- what a pass cannot do without ------------------------------------------------------

def _cells(case):
    return (2 * case["wake"] + 2 * case["surface"] - 2) * (case["normal"] - 1)


def _solve_work(cells, sst, mixed, iterations):
    # every geometry array, the state in and the state out once a pass;
    # operations: the assembled stages, and the pressure solve's iterations (a
    # CG iteration is 21 a cell; a mixed one about 150 with its V-cycle)
    arrays = 18 + (20 if sst else 13)
    per_cell = (1100 if sst else 600) + (16 * 150 if mixed else 200 * 21)
    return dict(bytes=8.0 * arrays * cells, flops=float(iterations) * per_cell * cells)


def work(case):
    kind = case["kind"]
    if kind == "solve":
        return _solve_work(_cells(case), case["model"] == "sst", case["precision"] == "mixed", case["iterations"])
    if kind == "batch":
        cells = case["points"] * _cells(case) + (192 * 48 + 384 * 96 if case["trio"] else 0)
        return _solve_work(cells, True, case["precision"] == "mixed", case["iterations"])
    if kind == "cg":
        n = case["cells_i"] * case["cells_j"]
        expected = min(case["cap"], 200 if case["tolerance"] >= 0.01 else case["cap"])
        return dict(bytes=8.0 * 5 * n, flops=21.0 * expected * n)
    if kind == "forces":
        stations = 2 * case["surface"] - 2
        return dict(bytes=8.0 * 24 * stations, flops=60.0 * stations)
    if kind == "streamlines":
        points = case["seeds"] * case["max_steps"] * (2 if case["backwards"] else 1)
        return dict(bytes=16.0 * points, flops=300.0 * points)
    return _solve_work(case["requests"] * _cells(case), True, True, case["iterations"])


# ---- the same results from plain numpy in 64 bits ------------------------------------------

class _Geometry:
    """Face metrics of a mesh (reference face order) as flat numpy arrays."""

    def __init__(self, mesh, conditions):
        self.ni, self.nj, self.n = mesh.cells_i, mesh.cells_j, mesh.cells
        self.own = mesh.owner.astype(np.int64)
        nb = mesh.neighbour.astype(np.int64)
        self.inner = nb >= 0
        cut = (mesh.boundary == cb.FACE_WAKECUT) & (mesh.partner >= 0) & ~self.inner
        other = np.where(self.inner, nb, -1)
        other[cut] = self.own[mesh.partner[cut]]
        self.cut, self.linked = cut, other >= 0
        self.other = np.where(self.linked, other, self.own)
        centre, face = mesh.centroid.reshape(-1, 2), mesh.face_centre.reshape(-1, 2)
        self.s = mesh.face_normal.reshape(-1, 2) * mesh.face_area[:, None]
        self.normal = mesh.face_normal.reshape(-1, 2)
        to_own = np.hypot(*(centre[self.own] - face).T)
        to_other = np.hypot(*(centre[self.other] - face).T)
        self.w = np.where(self.linked, to_other / (to_own + to_other), 1.0)
        d = np.where(self.linked[:, None], centre[self.other], face) - centre[self.own]
        self.big_d = (self.s ** 2).sum(1) / (self.s * d).sum(1)
        self.t = self.s - d * self.big_d[:, None]
        self.vol = mesh.cell_area
        self.kind = conditions.kind
        self.bc, self.bc_p = conditions.velocity.reshape(-1, 2), conditions.pressure
        j_faces = self.ni * (self.nj + 1)
        f = np.arange(self.own.size)
        self.is_j = f < j_faces
        walls = np.flatnonzero(self.kind == cb.BC_NOSLIP_WALL)
        self.walls = walls
        self.dist = np.full(self.n, np.inf)
        for k in walls:
            self.dist = np.minimum(self.dist, np.hypot(*(centre - face[k]).T))

    def gather(self, values, minus=None):
        """Per cell: the faces' values summed on their owner, and for interior
        faces `minus` (default the same) taken off their neighbour."""
        out = np.bincount(self.own, values, self.n)
        m = (values if minus is None else minus)[self.inner]
        return out - np.bincount(self.other[self.inner], m, self.n)

    def face(self, phi):
        return self.w * phi[self.own] + (1 - self.w) * phi[self.other]

    def grad(self, phi_f):
        return np.stack([self.gather(self.s[:, a] * phi_f) / self.vol for a in (0, 1)])


def _sweep_in_cell_order(g, diag, coef, b, x, sweeps):
    """Gauss-Seidel in cell order, one anti-diagonal of cells at a time."""
    ni, nj = g.ni, g.nj
    south, north, west, east, wake = coef
    for _ in range(sweeps):
        for d in range(ni + nj - 1):
            j = np.arange(max(0, d - ni + 1), min(nj - 1, d) + 1)
            i = d - j
            c = j * ni + i
            off = south[c] * x[np.maximum(c - ni, 0)] + north[c] * x[np.minimum(c + ni, g.n - 1)]
            off += west[c] * x[np.maximum(c - 1, 0)] + east[c] * x[np.minimum(c + 1, g.n - 1)]
            if j[0] == 0:
                off[0] += wake[i[0]] * x[ni - 1 - i[0]]
            x[c] = (b[c] - off) / diag[c]
    return x


def _rows(g, upper, lower):
    """S, N, W, E and wake coefficients per cell from face coefficients: upper
    on the owner's row, lower on the neighbour's."""
    south, north, west, east = (np.zeros(g.n) for _ in range(4))
    wake = np.zeros(g.ni)
    j_in, i_in = g.inner & g.is_j, g.inner & ~g.is_j
    north[g.own[j_in]], south[g.other[j_in]] = upper[j_in], lower[j_in]
    east[g.own[i_in]], west[g.other[i_in]] = upper[i_in], lower[i_in]
    wake[g.own[g.cut]] = upper[g.cut]
    return south, north, west, east, wake


def _cg(apply, diag, b, tolerance, cap):
    """Jacobi-preconditioned CG, L1 stopping rule: x, iterations, norms."""
    x = np.zeros_like(b)
    r = b.copy()
    first = last = np.abs(r).sum()
    z = r / diag
    d, rz, n = z.copy(), r @ z, 0
    while n < cap:
        q = apply(d)
        step = rz / (d @ q)
        x += step * d
        r -= step * q
        n, last = n + 1, np.abs(r).sum()
        if last <= tolerance * first:
            break
        z = r / diag
        rz, old = r @ z, rz
        d = z + (rz / old) * d
    return x, n, first, last


class _Simple:
    """The steady SIMPLE iteration (and k-omega SST) on flat numpy arrays."""

    def __init__(self, mesh, conditions, settings, field, sst):
        self.g, self.set, self.sst = _Geometry(mesh, conditions), settings, sst
        g = self.g
        self.u, self.v, self.p, self.rho, self.mol = (np.array(a, float) for a in field)
        self.mu = self.mol.copy()
        speed = np.hypot(self.u, self.v).max()
        far = g.kind == cb.BC_FARFIELD
        self.dead = np.where(far, 1e-3 * self.rho[g.own] * speed * np.hypot(*g.s.T), 0.0)
        self.mf = np.zeros(g.own.size)
        imposed = self._imposed()
        fu, fv = (np.where(g.linked, g.face(a), np.where(imposed, g.bc[:, k], a[g.own]))
                  for k, a in enumerate((self.u, self.v)))
        self.mf = np.where(g.inner, g.face(self.rho), self.rho[g.own]) * (fu * g.s[:, 0] + fv * g.s[:, 1])
        edge = ~g.inner & (g.kind != cb.BC_INTERNAL)
        self.ref = np.maximum(-self.mf[edge], 0).sum()
        if sst:
            self.k_in = 1.5 * (max(settings.inflow_intensity, 1e-8) * speed) ** 2
            self.w_in = max(self.rho.max() * self.k_in / (settings.inflow_viscosity_ratio * self.mu.max()), 1e-10)
            self.k, self.om = np.full(g.n, self.k_in), np.full(g.n, self.w_in)
            self.om = np.maximum(self.om, self._wall_omega(self.mol / self.rho, self.k))
            self.mut = self.rho * self.k / self.om
            self.mu = self.mol + self.mut

    def _imposed(self):
        g = self.g
        return ((g.kind == cb.BC_NOSLIP_WALL) | (g.kind == cb.BC_INLET)
                | ((g.kind == cb.BC_FARFIELD) & (self.mf < self.dead)))

    def _wall_omega(self, nu, k):
        d = np.maximum(self.g.dist, 1e-30)
        return np.hypot(6 * nu / (0.075 * d * d), np.sqrt(np.maximum(k, 0)) / (0.09 ** 0.25 * 0.41 * d))

    def iterate(self):
        g, st = self.g, self.set
        own, oth, inner, linked = g.own, g.other, g.inner, g.linked
        edge, imposed = ~linked, self._imposed()
        fu, fv = (np.where(linked, g.face(a), np.where(imposed, g.bc[:, k], a[own]))
                  for k, a in enumerate((self.u, self.v)))
        fp = np.where(linked, g.face(self.p), np.where(imposed, self.p[own], g.bc_p))
        gu, gv, gp = g.grad(fu), g.grad(fv), g.grad(fp)
        speed = np.hypot(self.u, self.v).max() or 1.0
        # momentum: upwind convection, over-relaxed diffusion, explicit cross terms
        vis = np.where(linked, g.face(self.mu), self.mu[own])
        dif = vis * g.big_d
        out, into = np.maximum(self.mf, 0), np.maximum(-self.mf, 0)
        at_edge = np.where(imposed, dif, self.mf)
        diag = np.bincount(own, np.where(linked, out + dif, at_edge), g.n)
        diag += np.bincount(oth[inner], (into + dif)[inner], g.n)
        upper, lower = np.where(linked, -into - dif, 0.0), np.where(inner, -out - dif, 0.0)
        sources = []
        for a, grad, phi, k in ((self.u, gu, gp[0], 0), (self.v, gv, gp[1], 1)):
            cross = st.non_orthogonal_blend * vis * (g.face(grad[0]) * g.t[:, 0] + g.face(grad[1]) * g.t[:, 1])
            fixed = (dif - self.mf) * g.bc[:, k] + st.non_orthogonal_blend * vis * (
                grad[0][own] * g.t[:, 0] + grad[1][own] * g.t[:, 1])
            term = np.where(linked, cross, np.where(imposed, fixed, 0.0))
            if st.scheme:
                ahead = self.mf * (g.face(a) - np.where(self.mf >= 0, a[own], a[oth]))
                term = np.where(inner, term - ahead, term)
            sources.append(g.gather(term) - phi * g.vol)
        relaxed = diag / st.velocity_relaxation
        sources = [b + (relaxed - diag) * a for b, a in zip(sources, (self.u, self.v))]
        diag = relaxed

        def off(x):
            s = np.bincount(own[linked], (upper * x[oth])[linked], g.n)
            return s + np.bincount(oth[inner], (lower * x[own])[inner], g.n)

        scale = np.abs(diag).sum() * speed
        res = [np.abs(b - diag * a - off(a)).sum() / scale for b, a in zip(sources, (self.u, self.v))]
        c = np.arange(g.n)
        colour = (c % g.ni + c // g.ni) & 1
        for _ in range(st.momentum_sweeps):
            for half in (0, 1):
                pick = colour == half
                for a, b in zip((self.u, self.v), sources):
                    a[pick] = ((b - off(a)) / diag)[pick]
        # Rhie-Chow fluxes and the pressure correction
        rho_f = np.where(linked, g.face(self.rho), self.rho[own])
        ratio = g.vol / diag
        mob = np.where(linked, g.face(ratio), ratio[own])
        imposed = self._imposed()
        flow = [np.where(linked, g.face(a), a[own]) for a in (self.u, self.v)]
        smooth = sum(np.where(linked, g.face(q), q[own]) * g.s[:, k] for k, q in enumerate(gp))
        jump = np.where(linked, self.p[oth], g.bc_p) - self.p[own]
        free = rho_f * (flow[0] * g.s[:, 0] + flow[1] * g.s[:, 1]) - rho_f * mob * (jump * g.big_d - smooth)
        fixed = rho_f * (g.bc[:, 0] * g.s[:, 0] + g.bc[:, 1] * g.s[:, 1])
        self.mf = np.where(edge & imposed, fixed, free)
        imposed = self._imposed()
        net = g.gather(self.mf)
        coef = np.where(edge & imposed, 0.0, rho_f * mob * g.big_d)
        p_diag = np.bincount(own, coef, g.n) + np.bincount(oth[inner], coef[inner], g.n)
        link = np.where(linked, coef, 0.0)

        def apply(x):
            y = p_diag * x - np.bincount(own, link * x[oth], g.n)
            return y - np.bincount(oth[inner], (link * x[own])[inner], g.n)

        x, count, _, _ = _cg(apply, p_diag, -net, st.pressure_tolerance, st.pressure_iterations)
        fx = np.where(linked, g.face(x), np.where(imposed, x[own], 0.0))
        gx = g.grad(fx)
        self.p = self.p + st.pressure_relaxation * x
        self.u = self.u - gx[0] * ratio
        self.v = self.v - gx[1] * ratio
        self.mf = self.mf - coef * (np.where(linked, x[oth], 0.0) - x[own])
        total = np.abs(net).sum()
        div = np.abs(g.gather(self.mf / self.rho[own]) / g.vol).max()
        monitor = [total / self.ref, res[0], res[1], total, div, float(count)] + [0.0] * 10
        if self.sst:
            monitor[6:] = self._turbulence(gu, gv)
        return np.array(monitor)

    def _turbulence(self, gu, gv):
        g, st, tiny = self.g, self.set, 1e-30
        own, oth, inner, linked = g.own, g.other, g.inner, g.linked
        s12 = 0.5 * (gu[1] + gv[0])
        strain = np.sqrt(2 * (gu[0] ** 2 + gv[1] ** 2 + 2 * s12 ** 2))
        wall = g.kind == cb.BC_NOSLIP_WALL
        inflow = ~linked & ((g.kind == cb.BC_INLET) | ((g.kind == cb.BC_FARFIELD) & (self.mf < 0)))
        w1 = np.where(inner, g.w, 1.0)
        grads = []
        for phi, at_wall, inlet in ((self.k, 0.0, self.k_in), (self.om, None, self.w_in)):
            f = w1 * phi[own] + (1 - w1) * phi[oth]
            f = np.where(inflow, inlet, f)
            grads.append(g.grad(f if at_wall is None else np.where(wall, at_wall, f)))
        gk, gw = grads
        d, nu = np.maximum(g.dist, tiny), self.mol / self.rho
        om, k = np.maximum(self.om, 1e-10), np.maximum(self.k, 0)
        cross = 2 * self.rho * 0.856 * (gk[0] * gw[0] + gk[1] * gw[1]) / om
        a = np.sqrt(k) / (0.09 * om * d)
        b = 500 * nu / (d * d * om)
        arg1 = np.minimum(np.maximum(a, b), 4 * self.rho * 0.856 * k / (np.maximum(cross, 1e-10) * d * d))
        f1 = np.tanh(np.clip(arg1 ** 4, 0, 50))
        f2 = np.tanh(np.clip(np.maximum(2 * a, b) ** 2, 0, 50))
        prod = np.minimum(self.mut * strain ** 2, 10 * 0.09 * self.rho * k * om)

        def blend(near, away):
            return f1 * near + (1 - f1) * away

        dt = np.abs(g.big_d)
        relax = min(max(st.turbulence_relaxation, 0.05), 1.0)
        g1 = 0.075 / 0.09 - 0.5 * 0.41 ** 2 / math.sqrt(0.09)
        g2 = 0.0828 / 0.09 - 0.856 * 0.41 ** 2 / math.sqrt(0.09)
        out, into = np.maximum(self.mf, 0), np.maximum(-self.mf, 0)
        result, norms = [], []
        for phi, sigma, at_wall, inlet, source, sink in (
                (self.k, blend(0.85, 1.0), 0.0, self.k_in, prod, 0.09 * self.rho * om),
                (self.om, blend(0.5, 0.856), self.w_in, self.w_in,
                 blend(g1, g2) * self.rho * strain ** 2 + (1 - f1) * cross, blend(0.075, 0.0828) * self.rho * om)):
            eff = self.mol + sigma * self.mut
            dif = (w1 * eff[own] + (1 - w1) * eff[oth]) * dt
            held = ~linked & (wall | inflow)
            value = np.where(wall, at_wall, inlet)
            diag = np.bincount(own, np.where(linked | held, dif, 0.0) + out, g.n)
            diag += np.bincount(oth[inner], (into + dif)[inner], g.n)
            rhs = np.bincount(own, np.where(held, (dif + into) * value, 0.0), g.n) + source * g.vol
            diag += sink * g.vol
            rhs += (diag / relax - diag) * phi
            diag = diag / relax
            coef = _rows(g, np.where(linked, -into - dif, 0.0), np.where(inner, -out - dif, 0.0))
            y = diag * phi
            y += np.bincount(own[linked], ((-into - dif) * phi[oth])[linked], g.n)
            y += np.bincount(oth[inner], ((-out - dif) * phi[own])[inner], g.n)
            norms.append(np.abs(rhs - y).sum() / max(np.abs(diag).sum() * max(inlet, tiny), 1e-300))
            result.append(_sweep_in_cell_order(g, diag, coef, rhs, phi.copy(), 3))
        self.k, self.om = np.maximum(result[0], 0), np.maximum(result[1], 1e-10)
        cells = np.unique(own[g.walls])
        self.om[cells] = self._wall_omega(nu, self.k)[cells]
        o, n = own[g.walls], -g.normal[g.walls]
        dn = self.u[o] * n[:, 0] + self.v[o] * n[:, 1]
        slip = np.hypot(self.u[o] - n[:, 0] * dn, self.v[o] - n[:, 1] * dn)
        yplus = np.sqrt(self.mol[o] * slip / d[o] / self.rho[o]) * d[o] / nu[o]
        self.mut = self.rho * 0.31 * self.k / np.maximum(np.maximum(0.31 * self.om, strain * f2), tiny)
        self.mu = self.mol + self.mut
        return [norms[0], norms[1], self.k.min(), self.k.max(), self.om.min(), self.om.max(), self.mut.min(),
                self.mut.max(), (self.mut / self.mol).max(), max(0.0, yplus.max())]


def _exact_solve(case, seed):
    mesh = _case_mesh(case)
    alpha, field = _start(mesh, case["alpha"], case["reynolds"], seed)
    s = _Simple(mesh, cb.freestream_conditions(mesh, 1.0, alpha), _settings(case), field, case["model"] == "sst")
    for _ in range(case["iterations"]):
        monitor = s.iterate()
    out = dict(U=s.u, V=s.v, P=s.p, monitor=monitor)
    if case["model"] == "sst":
        out.update(K=s.k, OMEGA=s.om, MUT=s.mut)
    return out


def _exact_cg(case, seed):
    diag, upper, source, across = _cg_arrays(case, seed)
    ni, nj = case["cells_i"], case["cells_j"]
    north = upper[:ni * (nj + 1)].reshape(nj + 1, ni)
    east = np.ascontiguousarray(upper[ni * (nj + 1):].reshape(ni + 1, nj).T)
    pair = np.where(across >= 0, across, 0)

    def apply(flat):
        x = flat.reshape(nj, ni)
        y = diag.reshape(nj, ni) * x
        y[1:] += north[1:-1] * x[:-1]
        y[:-1] += north[1:-1] * x[1:]
        y[:, 1:] += east[:, 1:-1] * x[:, :-1]
        y[:, :-1] += east[:, 1:-1] * x[:, 1:]
        y[0] += np.where(across >= 0, north[0] * x[0][pair], 0.0)
        return y.ravel()

    x, n, first, last = _cg(apply, diag, source, case["tolerance"], case["cap"])
    return dict(x=x, report=np.array([float(n), first, last]), converged=int(last <= case["tolerance"] * first))


def _exact_forces(case, seed):
    """Wall pressure and shear at the stations, and their integrals."""
    mesh = _case_mesh(case)
    alpha, field = _start(mesh, case["alpha"], case["reynolds"], seed)
    u, v, p = _developed(mesh, alpha, seed)
    mu = field[4]
    ni = mesh.cells_i
    face = np.flatnonzero(mesh.boundary[:ni] == cb.FACE_WALL)
    nodes = mesh.nodes.reshape(-1, 2)
    along = nodes[face + 1] - nodes[face]
    length = np.hypot(*along.T)
    tangent = along / length[:, None]
    own = mesh.owner[face]
    normal = -mesh.face_normal.reshape(-1, 2)[face]
    centre = mesh.face_centre.reshape(-1, 2)[face]
    cells = mesh.centroid.reshape(-1, 2)
    second = own + ni  # the cell above, along the wall normal on a C-grid
    d1, d2 = (np.abs(((cells[c] - centre) * normal).sum(1)) for c in (own, second))
    lead, stag = int(np.argmin(nodes[face][:, 0])), int(np.argmax(p[own]))
    k = np.arange(face.size)
    forward = np.where(k == stag, k >= lead, k > stag)
    flow = np.where(forward[:, None], tangent, -tangent)

    def slip(c):
        vel = np.stack([u[c], v[c]], 1)
        vel = vel - normal * (vel * normal).sum(1)[:, None]
        return (vel * flow).sum(1)

    u1, u2 = slip(own), slip(second)
    two = d2 > 1.05 * d1
    slope = np.where(two, (u1 * d2 ** 2 - u2 * d1 ** 2) / np.where(two, d1 * d2 * (d2 - d1), 1.0), u1 / d1)
    shear = mu[own] * slope
    push = normal * (-(p[own]) * length)[:, None]
    drag = flow * (shear * length)[:, None]
    wind = np.array([math.cos(math.radians(alpha)), math.sin(math.radians(alpha))])
    up = np.array([-wind[1], wind[0]])
    arm = centre - np.array([0.25, 0.0])
    both = push + drag
    moment = -(arm[:, 0] * both[:, 1] - arm[:, 1] * both[:, 0]).sum()
    q = 0.5
    order = np.concatenate([np.arange(lead, face.size), np.arange(lead - 1, -1, -1)])
    total = both.sum(0)
    return dict(coefficients=np.array([total @ up, total @ wind, moment, push.sum(0) @ wind, drag.sum(0) @ wind]) / q,
                cp=(p[own] / q)[order], cf=(shear / q)[order], stations=None)


def _exact_streamlines(case, seed):
    """RK4 through the cells' velocities, every curve a step at a time."""
    mesh = _case_mesh(case)
    alpha, _ = _start(mesh, case["alpha"], case["reynolds"], seed)
    u, v, _ = _developed(mesh, alpha, seed)
    ni, nj = mesh.cells_i, mesh.cells_j
    nodes = mesh.nodes.reshape(nj + 1, ni + 1, 2)
    ring = np.stack([nodes[:-1, :-1], nodes[:-1, 1:], nodes[1:, 1:], nodes[1:, :-1]], 2).reshape(-1, 4, 2)
    edge = np.roll(ring, -1, axis=1) - ring
    c = np.arange(mesh.cells)
    i, j = c % ni, c // ni
    across = np.full(ni, -1)
    cut = np.flatnonzero((mesh.boundary[:ni] == cb.FACE_WAKECUT) & (mesh.partner[:ni] >= 0))
    across[cut] = mesh.owner[mesh.partner[cut]]
    step_to = np.stack([np.where(j > 0, c - ni, across[i]), np.where(i < ni - 1, c + 1, -1),
                        np.where(j < nj - 1, c + ni, -1), np.where(i > 0, c - 1, -1)], 1)

    def beyond(cell, at):
        q = at[:, None, :] - ring[cell]
        return -(edge[cell, :, 0] * q[:, :, 1] - edge[cell, :, 1] * q[:, :, 0])

    def locate(at, cell):
        cell = cell.copy()
        moving = np.flatnonzero(cell >= 0)
        while moving.size:
            far = beyond(cell[moving], at[moving])
            worst = far.argmax(1)
            out = far[np.arange(moving.size), worst] > 0
            moving, worst = moving[out], worst[out]
            cell[moving] = step_to[cell[moving], worst]
            moving = moving[cell[moving] >= 0]
        return cell

    seeds = _seeds(case, seed)
    start = np.array([np.append(np.flatnonzero((beyond(c, np.repeat(s[None], c.size, 0)) <= 0).all(1)), -1)[0]
                      for s in seeds])
    halves = []
    for sense in ((-1.0, 1.0) if case["backwards"] else (1.0,)):
        curves = [[s] if k >= 0 else [] for s, k in zip(seeds, start)]
        live = np.flatnonzero(start >= 0)
        at, cell = seeds[live].copy(), start[live]
        for _ in range(case["max_steps"]):
            def speed_at(where, hint):
                found = locate(where, hint)
                vel = np.where((found >= 0)[:, None], np.stack([u[found], v[found]], 1) * sense, 0.0)
                return vel, np.where(found >= 0, found, hint)
            k1, h = speed_at(at, cell)
            speed = np.hypot(*k1.T)
            go = speed > 1e-4
            live, at, cell, k1, h, speed = live[go], at[go], cell[go], k1[go], h[go], speed[go]
            if not live.size:
                break
            dt = (0.35 * np.sqrt(mesh.cell_area[cell]) / speed)[:, None]
            k2, h = speed_at(at + k1 * (0.5 * dt), h)
            k3, h = speed_at(at + k2 * (0.5 * dt), h)
            k4, h = speed_at(at + k3 * dt, h)
            at = at + (k1 + 2 * k2 + 2 * k3 + k4) * (dt / 6)
            cell = locate(at, cell)
            go = cell >= 0
            live, at, cell = live[go], at[go], cell[go]
            for k, xy in zip(live, at):
                curves[k].append(xy)
        halves.append(curves)
    if len(halves) == 1:
        halves.insert(0, [[] for _ in seeds])
    points = []
    for back, ahead in zip(*halves):
        if len(back) + len(ahead) >= 4:
            points += back[::-1] + ahead[1:]
    vertices = np.zeros((_vertices(case), 2))
    vertices[:len(points)] = np.array(points).reshape(-1, 2)
    return dict(lengths=None, vertices=vertices)


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve" and case["precision"] == "plain":
        return _exact_solve(case, seed)
    if kind == "cg":
        return _exact_cg(case, seed)
    if kind == "forces":
        return _exact_forces(case, seed)
    if kind == "streamlines":
        return _exact_streamlines(case, seed)
    # the mixed form stops its pressure solves at a tolerance of its own, and
    # a batch or a serving run takes numpy minutes
    return None
