"""Wall distances of a mesh in very large and very small units: a mesh scaled by
a power of two has its distances scaled exactly, also where the squares of its
coordinates leave FP32's range."""
import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d
from gpueularsolver2d_gb300 import _lib

pytestmark = pytest.mark.gpu


def distances(x, y, tri, scale):
    mesh = e2d.Mesh.from_arrays(x * scale, y * scale, tri)
    d = np.zeros(mesh.info(2.0 * scale).ncell)
    _lib.check(_lib.load().e2d_wall_distance(mesh._h, 2.0 * scale, d.ctypes.data_as(_lib.ctypes.POINTER(_lib.ctypes.c_double))))
    return d


@pytest.mark.parametrize("power", [-100, -70, -30, 30, 49, 60, 64, 66, 100, 200])
def test_scaled_mesh(lib, power):
    x, y, tri = e2d.Mesh.ogrid(96, 24, seed=3).nodes()
    assert np.array_equal(distances(x, y, tri, 2.0 ** power), distances(x, y, tri, 1.0) * 2.0 ** power)
