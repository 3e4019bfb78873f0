"""The plain form's solves on teams of CTAs: blocks whose row sweeps take 1 to
4 cells per lane with a full or a short last chunk, more chunks than a CTA has
warps, more rows than a sweep keeps edges of, teams too small for one sweep per
CTA, and several solves sharing one launch.

One outer iteration is compared with the CPU oracle: only the pressure CG's
sums run in another order, which moves the fields by rounding times the CG's
growth; 1e-9 of the field's scale is allowed, as for the stages. How many CTAs
work on a solve must not move a bit."""
import numpy as np
import pytest

import cfd_b200 as cb
from helpers import BaselineCase, rel_err
from oracle import port

pytestmark = pytest.mark.gpu

FIELDS = {"U": 0, "V": 1, "P": 2, "MASS_FLUX": 5, "K": 22, "OMEGA": 23, "MUT": 24}
# (surface, wake, normal): cells 2 * (surface + wake) - 2 by normal - 1
GRIDS = [(20, 8, 6), (100, 29, 12), (100, 30, 7), (70, 30, 200), (200, 58, 11), (300, 86, 9), (400, 114, 8),
         (800, 227, 7)]
SHORT = [(20, 8, 6), (70, 30, 200), (200, 58, 11), (400, 114, 8)]


def _mesh(grid):
    surface, wake, normal = grid
    return cb.cgrid("0012", surface_points=surface, wake_points=wake, normal_points=normal, first_layer_height=1e-4)


def _packed():
    BaselineCase("c2")
    return BaselineCase._golden["c2/settings"]


def _solver(mesh, alpha=3.0, model=2):
    p = _packed()
    s = cb.SimpleSolver.create(mesh, cb.freestream_conditions(mesh, 1.0, alpha),
                               cb.Settings.defaults(inflow_intensity=p[7], inflow_viscosity_ratio=p[8]))
    s.set_turbulence_model(model)
    s.initialise(*cb.uniform_field(mesh, 1.0, alpha, 1.0, 1e6))
    return s


def _fields(solver):
    return {f: solver.read(f) for f in FIELDS}


@pytest.mark.parametrize("grid", GRIDS)
def test_first_iteration_matches_the_oracle(grid):
    mesh = _mesh(grid)
    o = port.OracleSolver(mesh, cb.freestream_conditions(mesh, 1.0, 3.0), _packed(), 2, port.DEVICE_ORDER)
    o.initialise(*cb.uniform_field(mesh, 1.0, 3.0, 1.0, 1e6))
    o.iterate(1)
    s = _solver(mesh)
    s.iterate(1)
    for f, a in _fields(s).items():
        assert rel_err(a, o.read(FIELDS[f])) <= 1e-9, (f, rel_err(a, o.read(FIELDS[f])))


@pytest.mark.parametrize("grid", SHORT)
def test_the_bits_do_not_depend_on_the_team(grid, monkeypatch):
    mesh = _mesh(grid)
    alone = _solver(mesh)
    alone.iterate(3)
    want = _fields(alone)
    for ctas in (1, 3, 5, 16):
        monkeypatch.setenv("CFD_CLUSTER_SIZE", str(ctas))
        s = _solver(mesh)
        s.iterate(3)
        for f, a in _fields(s).items():
            assert np.array_equal(a, want[f]), (ctas, f)


@pytest.mark.parametrize("count", [3, 40, 160])
def test_solves_that_share_a_launch_keep_their_bits(count):
    meshes = [_mesh(g) for g in ((20, 8, 6), (100, 30, 7), (40, 12, 30))]
    make = lambda k: _solver(meshes[k % 3], alpha=float(k % 5), model=0 if k % 7 == 3 else 2)  # noqa: E731
    solvers = [make(k) for k in range(count)]
    batch = cb.Batch(solvers)
    batch.iterate(2)
    for k in range(0, count, max(1, count // 12)):
        alone = make(k)
        alone.iterate(2)
        a, b = _fields(solvers[k]), _fields(alone)
        for f in FIELDS:
            assert np.array_equal(a[f], b[f]), (k, f)
