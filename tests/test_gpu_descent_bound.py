"""A degenerate tree -- every face the same triangle, so every box meets every query -- ends a descent at its bound with
YS_FLAG_STACK_OVF, and below the bound every face is a row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STACK_OVF = 2


def _spec(faces):
    from ysim_b200 import _lib, generators as G
    spec = G.config_c1(P=6, level=1)
    cloth, obst = spec.meshes
    cloth.x = cloth.x + np.float32([0, 2, -2])  # inside the triangle's box, well off its plane
    obst.x = np.float32([[-5, -5, -5], [5, -5, -5], [0, 5, 5]])
    obst.v = obst.mass = obst.mask = None
    obst.facets = np.tile(np.uint32([0, 1, 2]), (faces, 1))
    assert obst.flags & _lib.MESH_STATIC
    return spec


# two vertices per warp share 2 x 2^18 steps: a face is a candidate of both and every 32nd one more run
@pytest.mark.parametrize("faces,stops", [(100000, False), (270000, True)])
def test_stack_flag(cuda_lib, faces, stops):
    from ysim_b200.scene import Scene
    s = Scene(_spec(faces))
    try:
        s.step(1)
        st = s.stats()
        assert bool(st["flags"] & STACK_OVF) == stops
        assert st["contacts"] == 0
        if stops:
            assert st["broad_rows"] < s.spec.meshes[0].nV * faces
        else:
            assert st["broad_rows"] == s.spec.meshes[0].nV * faces
    finally:
        s.close()
