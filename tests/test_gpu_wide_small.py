"""The CG primitive on systems so small that their inner products are subnormal."""
import numpy as np
import pytest

from test_gpu_wide_cg import TOL, _block, _device, _numpy_cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noalloc", [False, True])
def test_an_inner_product_without_a_reciprocal(noalloc):
    # r.z = 4e-309 at the start: 1 / (r.z) is infinite, the quotients of such
    # products are not. A term of a sum is 2e-311, which rounds to 3e-13 of itself;
    # three iterations, so within the tolerance of the ordinary systems
    diag, north, east, b, across = _block(20, 10, None)
    b = b * np.sqrt(4e-309 / np.sum(b * b / diag))
    x0 = np.zeros_like(b)
    want, first, last = _numpy_cg(diag, north, east, b, across, x0, 3)
    got, report = _device(diag, north, east, b, across, x0, 3, noalloc)
    assert np.max(np.abs(want)) > 0.0
    assert np.max(np.abs(got - want)) <= TOL * np.max(np.abs(want))
    assert report[0] == 3 and report[1] == pytest.approx(first, rel=TOL)


@pytest.mark.parametrize("ni,nj", [(20, 10), (192, 48), (300, 90), (768, 40)])
def test_a_solve_that_runs_until_nothing_is_left(ni, nj):
    # tolerance 0: the inner products become subnormal, then zero, long after the
    # solution stands. Both solutions are within their rounding, ~1e-15 times the
    # system's condition (~1e2), of the true one
    diag, north, east, b, across = _block(ni, nj, None)
    x0 = np.random.default_rng(9).standard_normal(b.shape)
    want, _, _ = _numpy_cg(diag, north, east, b, across, x0, 300)
    got, report = _device(diag, north, east, b, across, x0, 5000)
    assert np.max(np.abs(got - want)) <= TOL * np.max(np.abs(want))
    assert 0 < report[0] <= 5000 and 0.0 <= report[2] < 1e-100
