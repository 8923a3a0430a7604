"""StructuredMaterial3D.get_values does not depend on how a range is cut: large
ranges, whose threads work several cells of a column, against planes, columns
and cells evaluated by themselves (one cell per thread), bit for bit."""
import numpy as np
import pytest

from test_structured import _random_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,polygons,circles", [(3, False, False), (11, True, False), (21, True, True)])
@pytest.mark.parametrize("shape", [(41, 31, 121), (41, 31, 130), (41, 31, 1937)])   # 2, 2 and 16 cells a thread
def test_large_ranges_equal_their_parts(seed, polygons, circles, shape):
    mat, _ = _random_layout(seed, n=12, polygons=polygons, circles=circles)
    nx, ny, nz = shape
    whole = mat.get_values(0, nx, 0, ny, -20, nz - 20, 0.5, 0.0, -0.5)
    for i in (0, 1, 15, 16, 17, 20, 25, 31, 32, 47, 48, nz - 17, nz - 1):
        assert np.array_equal(mat.get_values(0, nx, 0, ny, i - 20, i - 19, 0.5, 0.0, -0.5)[0], whole[i])
    for j, k in ((0, 0), (ny // 2, nx // 3), (ny - 1, nx - 1)):
        assert np.array_equal(mat.get_values(k, k + 1, j, j + 1, -20, nz - 20, 0.5, 0.0, -0.5)[:, 0, 0], whole[:, j, k])
