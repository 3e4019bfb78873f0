"""Batches whose plan matters: a captured graph beside changes of plan."""
import numpy as np
import pytest

import cfd_b200 as cb

pytestmark = pytest.mark.gpu

FIELDS = ("U", "V", "P", "MASS_FLUX", "K", "OMEGA", "MUT")
# (surface, wake, normal): 2 * (surface + wake) - 2 by normal - 1 cells, the grids
# of test_plans.SIX
GRIDS = [(168, 84, 56), (109, 54, 56), (237, 118, 133), (107, 53, 61), (102, 50, 186), (55, 27, 153)]


def _solver(grid, alpha, **settings):
    surface, wake, normal = grid
    mesh = cb.cgrid("0012", surface_points=surface, wake_points=wake, normal_points=normal, first_layer_height=1e-4)
    s = cb.SimpleSolver.create(mesh, cb.freestream_conditions(mesh, 1.0, alpha),
                               cb.Settings.defaults(inflow_viscosity_ratio=10.0, **settings))
    s.set_turbulence_model(cb.MODEL_SST)
    s.initialise(*cb.uniform_field(mesh, 1.0, alpha, 1.0, 1e6))
    return s


def test_a_graph_is_captured_again_when_the_plan_changes():
    # SST members that become laminar need another plan (other CTAs, other shared
    # memory); the graph's next replay must give what direct launches give
    laminar = (0, 4, 5)
    make = lambda: [_solver(g, 0.5 * k) for k, g in enumerate(GRIDS)]  # noqa: E731
    solvers = make()
    batch = cb.Batch(solvers)
    batch.graph_launch(1)
    batch.monitors()
    for k in laminar:
        solvers[k].set_turbulence_model(cb.MODEL_LAMINAR)
    batch.iterate(1)
    batch.graph_launch(1)
    taken, _ = batch.monitors()
    assert taken == [1] * len(solvers)
    alone = make()
    for k, s in enumerate(alone):
        s.iterate(1)
        if k in laminar:
            s.set_turbulence_model(cb.MODEL_LAMINAR)
        s.iterate(2)
        for f in FIELDS:
            assert np.array_equal(solvers[k].read(f), s.read(f)), (k, f)
    batch.close()


@pytest.mark.parametrize("precision,flag", [(0, 256), (1, 64)])  # waits that give up, for tests
def test_a_fault_is_kept_until_it_is_read(precision, flag, monkeypatch):
    # a later launch must not erase what an earlier one reported: a CTA may give up
    # before the first CTA of its solve has begun
    solvers = [_solver((55, 27, 20), 1.0, precision=precision) for _ in range(2)]
    batch = cb.Batch(solvers)
    monkeypatch.setenv("CFD_KERNEL_FLAGS", str(flag))
    batch.launch(1)
    monkeypatch.delenv("CFD_KERNEL_FLAGS")
    batch.launch(1)
    with pytest.raises(cb.CfdError) as err:
        batch.monitors()
    assert err.value.code == 8  # CFD_INTERNAL
    # read once, for every solve of the batch
    taken, last = batch.iterate(1)
    assert taken == [1, 1] and all(np.isfinite(m.continuity) for m in last)
    assert np.isfinite(solvers[1].iterate(1).continuity)
    batch.close()


def test_a_new_start_drops_an_unread_fault(monkeypatch):
    s = _solver((55, 27, 20), 1.0)
    batch = cb.Batch([s])
    monkeypatch.setenv("CFD_KERNEL_FLAGS", "256")
    batch.launch(1)
    monkeypatch.delenv("CFD_KERNEL_FLAGS")
    import torch
    torch.cuda.synchronize()
    s.initialise(*cb.uniform_field(s.mesh, 1.0, 1.0, 1.0, 1e6))
    assert np.isfinite(s.iterate(1).continuity)
    batch.close()


def test_a_wide_solve_waits_behind_a_long_narrow_one():
    # the plan gives solve 2 (490x73) to the 74 CTAs of which 12 first run solve 0
    # (50x94): the others wait in solve 2's first barrier for all of that, here
    # seconds, and must not give up
    import time
    narrow = dict(pressure_iterations=300, pressure_tolerance=0.0, non_orthogonal_correctors=120,
                  pressure_relaxation=0.01)
    make = lambda: ([_solver((17, 9, 95), float(k), **narrow) for k in range(2)] +  # noqa: E731
                    [_solver((164, 82, 74), float(k)) for k in range(2)])
    iterations = 32
    together, alone = make(), make()
    for s in together[2:] + alone[2:]:
        s.set_turbulence_model(cb.MODEL_LAMINAR)
    batch = cb.Batch(together)
    start = time.perf_counter()
    taken, _ = batch.iterate(iterations)
    assert time.perf_counter() - start > 2.0  # longer than any fixed second
    assert taken == [iterations] * 4
    for k in (0, 2, 3):
        s = alone[k]
        s.iterate(iterations)
        for f in FIELDS[:4]:
            assert np.array_equal(together[k].read(f), s.read(f)), (k, f)
    batch.close()
