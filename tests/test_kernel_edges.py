"""Kernels at the sizes where their tiling can go wrong: edges of tiles,
remainders, the smallest and largest of a dispatch rule's range."""

import numpy as np
import pytest

import kat_scenes as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [4, 5, 18, 33])
@pytest.mark.parametrize("mesh", ["cube", "sphere6x5", "torus21x11", "far", "nan"])
def test_bake_bricks_and_chunks(oracle, res, mesh):
    """Grids that are no multiple of a warp's brick against meshes of one
    chunk of triangles, a partial last chunk, far from the origin, and with a
    triangle whose corner is not a number: the oracle's field bit for bit."""
    from pfsim import mesh as M

    if mesh == "sphere6x5":
        v, i = K.uv_sphere(0.5, 6, 5)
    elif mesh == "torus21x11":
        v, i = K.torus(0.4, 0.12, 21, 11)
    else:
        v, i = K.unit_cube_mesh((0.3, 0.2, 0.45))
        if mesh == "far":
            v = (v + np.array([37.0, -5.0, 110.0], np.float32)).astype(np.float32)
        elif mesh == "nan":
            v = np.vstack([v, np.array([[np.nan, 0.0, 0.0]], np.float32)])
            i = np.concatenate([i, np.array([0, 1, len(v) - 1], np.uint32)])
    a = M.bake_sdf(v, i, res, 0.07)
    b = oracle.bake_sdf(v, i, res, 0.07)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2] == b[2] and a[3] == b[3]
