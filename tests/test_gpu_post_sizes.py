"""Wall forces and streamlines at sizes where their kernels' passes end: fewer
stations than a block's threads, as many, one pair more and several times as
many; one curve, and more curves than the GPU has SMs. Against the
framework-independent 64-bit results of the measured cases."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from perf import cases  # noqa: E402

pytestmark = pytest.mark.gpu


def _pair(case, seed):
    out, ref = cases.run(cases.prepare(case, seed)), cases.exact(case, seed)
    assert set(ref) <= set(out)
    return [(name, np.asarray(out[name]), np.asarray(ref[name])) for name in ref if ref[name] is not None]


# 2 * surface - 2 stations, 512 threads. Sums of up to 1,038 terms in 64 bits:
# 1e-13 a term's rounding accumulated, relative to the largest value
@pytest.mark.parametrize("surface", [9, 40, 256, 257, 258, 400, 520])
def test_forces_at_the_edges_of_a_block(surface):
    case = dict(kind="forces", section="2412", first_layer=1e-4, alpha=5.0, reynolds=1e6, surface=surface, wake=20,
                normal=15)
    for name, a, b in _pair(case, 3):
        assert a.shape == b.shape
        assert np.max(np.abs(a - b)) <= 1e-11 * max(1.0, np.max(np.abs(b))), name


# a curve's points are the same steps in the same order: rounding of hypot alone,
# which the steps of a curve carry on
@pytest.mark.parametrize("seeds,steps,backwards", [(1, 1, False), (1, 60, True), (7, 300, True), (160, 40, True)])
def test_streamlines_of_any_count(seeds, steps, backwards):
    case = dict(kind="streamlines", section="0012", first_layer=1e-4, alpha=3.0, reynolds=1e6, surface=40, wake=20,
                normal=30, seeds=seeds, max_steps=steps, backwards=backwards)
    for name, a, b in _pair(case, 5):
        assert a.shape == b.shape
        assert np.max(np.abs(a - b)) <= 1e-9, name
