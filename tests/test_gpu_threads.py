"""Lone solves advanced from several host threads at once: each launch takes a share
of the GPU by how many others are in flight, which must not move a bit."""
import threading

import numpy as np
import pytest

import cfd_b200 as cb
from test_gpu_wide_cg import _block, _device

pytestmark = pytest.mark.gpu

FIELDS = ("U", "V", "P", "MASS_FLUX", "K", "OMEGA", "MUT")
GRIDS = [(128, 65, 97), (64, 33, 49), (77, 41, 62), (256, 129, 60)]


def _solver(grid, alpha, precision):
    surface, wake, normal = grid
    mesh = cb.cgrid("0012", surface_points=surface, wake_points=wake, normal_points=normal, first_layer_height=1e-4)
    s = cb.SimpleSolver.create(mesh, cb.freestream_conditions(mesh, 1.0, alpha),
                               cb.Settings.defaults(inflow_viscosity_ratio=10.0, precision=precision))
    s.set_turbulence_model(cb.MODEL_SST)
    s.initialise(*cb.uniform_field(mesh, 1.0, alpha, 1.0, 1e6))
    return s


def _at_once(work, count):
    gate, failed = threading.Barrier(count), []

    def run(k):
        try:
            gate.wait()
            work(k)
        except Exception as e:  # noqa: BLE001
            failed.append(e)
    threads = [threading.Thread(target=run, args=(k,)) for k in range(count)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.mark.parametrize("precision", [0, 1])
def test_solves_of_several_threads_keep_their_bits(precision):
    make = lambda: [_solver(GRIDS[k % 4], float(k), precision) for k in range(8)]  # noqa: E731
    solvers, alone = make(), make()
    _at_once(lambda k: [solvers[k].iterate(2) for _ in range(4)], len(solvers))
    for k, s in enumerate(alone):
        s.iterate(8)
        for f in FIELDS:
            assert np.array_equal(solvers[k].read(f), s.read(f)), (k, f)


def test_cg_solves_of_several_threads_keep_their_bits():
    systems = [_block(*shape, None, seed=n) for n, shape in enumerate([(768, 192), (384, 96), (192, 48), (300, 90)] * 2)]
    start = [np.random.default_rng(n).standard_normal(s[3].shape) for n, s in enumerate(systems)]
    alone = [_device(*s, x, 200) for s, x in zip(systems, start)]
    got = [None] * len(systems)

    def work(k):
        for _ in range(3):
            got[k] = _device(*systems[k], start[k], 200)
    _at_once(work, len(systems))
    for (x, report), (want, first) in zip(got, alone):
        assert np.array_equal(x, want) and np.array_equal(report, first)
