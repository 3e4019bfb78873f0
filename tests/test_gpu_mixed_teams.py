"""The mixed form on teams of any width: a solve gives the same bits on any
number of CTAs (fewer than six run the k/omega sweeps one after another), with
the sweeps' rows chained across CTAs or not, with a V-cycle's half sweeps
formed together or each as a phase of its own, and beside other solves. On
grids where tiles and rows end raggedly: an odd number of rows (the top
aggregate row is half empty), rows shorter than a warp and longer than a
block's threads (2, 3 and 4 cells a thread), column counts that halve once or
not at all, one or no coarse level."""
import numpy as np
import pytest

import cfd_b200 as cb

pytestmark = pytest.mark.gpu

FIELDS = ("U", "V", "P", "MASS_FLUX", "K", "OMEGA", "MUT")
# surface, wake, normal points: (2 wake + 2 surface - 4 + 2) x (normal - 1) cells
GRIDS = {"22x7": (8, 4, 8), "70x12": (24, 12, 13), "234x61": (77, 41, 62), "384x96": (128, 65, 97),
         "766x33": (256, 128, 34)}


def _solve(grid, monkeypatch, iterations=2, flags=0, ctas=None, threads=None):
    monkeypatch.setenv("CFD_KERNEL_FLAGS", str(flags))
    for name, value in (("CFD_CLUSTER_SIZE", ctas), ("CFD_THREADS", threads)):
        if value is None:
            monkeypatch.delenv(name, raising=False)
        else:
            monkeypatch.setenv(name, str(value))
    s = _start(grid)
    _, hist = s.iterate(iterations, history=True)
    out = {f: s.read(f) for f in FIELDS}
    s.close()
    return out, hist


def _start(grid, alpha=4.0):
    surface, wake, normal = GRIDS[grid]
    mesh = cb.cgrid("0012", surface_points=surface, wake_points=wake, normal_points=normal, first_layer_height=1e-4,
                    upstream_chords=10.0, downstream_chords=15.0, vertical_chords=10.0)
    s = cb.SimpleSolver.create(mesh, cb.freestream_conditions(mesh, 1.0, alpha),
                               cb.Settings.defaults(inflow_viscosity_ratio=10.0, precision=1))
    s.set_turbulence_model(cb.MODEL_SST)
    s.initialise(*cb.uniform_field(mesh, 1.0, alpha, 1.0, 1e6))
    return s


def _same(a, b):
    assert np.all(np.isfinite(a[1])) and np.array_equal(a[1], b[1])
    for f in FIELDS:
        assert np.array_equal(a[0][f], b[0][f]), f


@pytest.mark.parametrize("ctas", [1, 2, 5, 6, 16])
@pytest.mark.parametrize("grid", list(GRIDS))
def test_the_bits_do_not_depend_on_the_team(grid, ctas, monkeypatch):
    _same(_solve(grid, monkeypatch), _solve(grid, monkeypatch, ctas=ctas))


@pytest.mark.parametrize("threads", [64, 192, 256, 512])
@pytest.mark.parametrize("grid", list(GRIDS))
def test_chained_rows_and_fused_half_sweeps_give_the_phased_bits(grid, threads, monkeypatch):
    # bit 5: the sweeps one after another on one CTA per equation; bit 9: the
    # V-cycle's half sweeps as phases of their own
    a = _solve(grid, monkeypatch, threads=threads)
    for flags in (32, 512):
        _same(a, _solve(grid, monkeypatch, flags=flags, threads=threads))


@pytest.mark.parametrize("sweeps", ["1,1,1", "2,1,2", "1,2,3", "3,2,1"])
def test_multigrid_sweep_counts_agree_fused_and_phased(sweeps, monkeypatch):
    monkeypatch.setenv("CFD_MG", sweeps)
    _same(_solve("234x61", monkeypatch), _solve("234x61", monkeypatch, flags=512))


def test_a_batch_gives_each_solve_its_own_bits(monkeypatch):
    # more cells than the GPU takes side by side at their widest: teams with
    # several solves each
    grids = ["384x96", "766x33", "234x61", "384x96", "22x7", "70x12", "384x96"]
    together = [_start(g, float(k)) for k, g in enumerate(grids)]
    batch = cb.Batch(together)
    batch.iterate(2)
    for k, g in enumerate(grids):
        alone = _start(g, float(k))
        alone.iterate(2)
        for f in FIELDS:
            assert np.array_equal(together[k].read(f), alone.read(f)), (k, f)
        alone.close()
    batch.close()


def test_a_chain_wait_that_gives_up_is_reported(monkeypatch):
    with pytest.raises(cb.CfdError) as err:
        _solve("384x96", monkeypatch, iterations=1, flags=64)
    assert err.value.code == 8  # CFD_INTERNAL
    assert "k/omega sweep stage" in str(err.value)
    _same(_solve("384x96", monkeypatch), _solve("384x96", monkeypatch, flags=32))
