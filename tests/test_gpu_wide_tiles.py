"""The pressure CG on blocks that are tiled in narrow column tiles: a width that
divides into them and one that leaves the last tile short, a last unit of fewer
rows, wake cuts whose partners lie in other tiles, and more rows than the GPU's
CTAs hold a unit each of."""
import pytest

from test_gpu_wide_cg import _block, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj,wake", [(302, 190, "row"), (642, 151, "row"), (766, 190, "row"), (768, 161, None),
                                        (65, 1433, None), (129, 600, None), (515, 433, None)])
def test_narrow_tiles(ni, nj, wake):
    _check(_block(ni, nj, wake))
