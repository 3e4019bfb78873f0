"""The plain form at the edges of its tiling, mostly on fewer than 512 threads: column counts that leave
fewer tiles than asked for at the width they get, and ordinary grids with threads
that do or do not fill a unit of the CG.

One outer iteration against the CPU oracle, with the tolerance of the 512-thread
tests: only the pressure CG's sums run in another order, which moves the fields by
rounding times the CG's growth; 1e-9 of the field's scale is allowed."""
import pytest

import cfd_b200 as cb
from helpers import rel_err
from oracle import port
from test_gpu_plain_teams import FIELDS, _fields, _mesh, _packed, _solver

pytestmark = pytest.mark.gpu

# threads, (surface, wake, normal): 2 * (surface + wake) - 2 columns
CASES = [(32, (900, 126, 7)), (64, (1300, 238, 7)), (128, (1300, 238, 12)), (32, (20, 8, 6)), (96, (70, 30, 60)),
         (160, (100, 29, 40)), (256, (200, 58, 30)), (288, (70, 30, 60)),
         (512, (800, 227, 41))]  # 17 chunks and 40 rows: a sweep's kept edges are used again


@pytest.mark.parametrize("threads,grid", CASES)
def test_first_iteration_matches_the_oracle(threads, grid, monkeypatch):
    monkeypatch.setenv("CFD_THREADS", str(threads))
    mesh = _mesh(grid)
    o = port.OracleSolver(mesh, cb.freestream_conditions(mesh, 1.0, 3.0), _packed(), 2, port.DEVICE_ORDER)
    o.initialise(*cb.uniform_field(mesh, 1.0, 3.0, 1.0, 1e6))
    o.iterate(1)
    s = _solver(mesh)
    s.iterate(1)
    for f, a in _fields(s).items():
        assert rel_err(a, o.read(FIELDS[f])) <= 1e-9, (f, rel_err(a, o.read(FIELDS[f])))


@pytest.mark.parametrize("wake,normal", [(52170, 4), (52186, 4), (60000, 3)])
def test_very_wide_blocks(wake, normal):
    # 104,418 columns: a sweep's chunk edges just fit on chip; 104,450 and more: none
    # are kept there
    mesh = cb.cgrid("0012", surface_points=40, wake_points=wake, normal_points=normal, first_layer_height=1e-3)
    o = port.OracleSolver(mesh, cb.freestream_conditions(mesh, 1.0, 3.0), _packed(), 2, port.DEVICE_ORDER)
    o.initialise(*cb.uniform_field(mesh, 1.0, 3.0, 1.0, 1e6))
    o.iterate(1)
    s = _solver(mesh)
    s.iterate(1)
    for f, a in _fields(s).items():
        assert rel_err(a, o.read(FIELDS[f])) <= 1e-9, (f, rel_err(a, o.read(FIELDS[f])))
