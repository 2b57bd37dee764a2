"""Staged calls out of their order: narrow before any detect works on no rows, update before any narrow on no contacts,
and the rows of a fused substep, which stores none, are not taken for a detect's."""
import numpy as np
import pytest

from tests.test_gpu_groups import _folded

pytestmark = pytest.mark.gpu


def _apart():
    """A cloth well above its obstacle."""
    spec = _folded(12, 0)
    spec.meshes[0].x = spec.meshes[0].x + np.float32([0, 1, 0])
    return spec


def test_update_first(cuda_lib):
    from ysim_b200.scene import Scene
    a, b = Scene(_apart()), Scene(_apart())
    try:
        a.system.snapshot_xprev()
        a.system.update()
        b.step_staged(1)
        for w in ("x", "v", "xprev"):
            assert np.array_equal(a.get(w).view(np.uint32), b.get(w).view(np.uint32))
        assert a.stats()["flags"] == b.stats()["flags"] == 0
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("detected", [False, True], ids=["fresh", "after_detect"])
def test_narrow_without_rows(cuda_lib, detected):
    from ysim_b200.scene import Scene
    s = Scene(_folded(20, 1))
    try:
        if detected:
            s.step_staged(2)
            assert len(s.rows()) > 0
        s.step(2)
        assert s.stats()["broad_rows"] > 0 and len(s.rows()) == 0
        s.narrow_phase.narrow_and_sort_by_vertices()
        off, c = s.contacts()
        assert len(c) == 0 and not off.any()
        s.broad_phase.refit_swept()
        s.broad_phase.detect_collisions()
        assert len(s.rows()) > 0
    finally:
        s.close()
