"""Staged calls after a fused substep: they read the trees, root boxes and grid extents of that substep's refit, as they
do after a staged substep (the two paths leave the same state, so every comparison is exact)."""
import numpy as np
import pytest

from tests.helpers import canon_rows_full
from tests.test_gpu_groups import _folded
from ysim_b200.scene import W4_EMPTY

pytestmark = pytest.mark.gpu

LAYOUTS = {"reference": 0, "cube": 1}


def _pair(spec, layout, steps):
    """The same scene after `steps` substeps, the last of them (fused, staged)."""
    from ysim_b200.scene import Scene
    out = []
    for staged in (False, True):
        s = Scene(spec, tree_layout=LAYOUTS[layout])
        s.step(steps - 1)
        s.step_staged(1) if staged else s.step(1)
        out.append(s)
    for w in ("x", "v", "xprev"):
        assert np.array_equal(out[0].get(w), out[1].get(w))
    return out


def _drop(steps):
    """A grid cloth without self rows that comes down on its obstacle: only its root box is refit, and the box of its
    start does not meet the obstacle's."""
    from ysim_b200 import generators as G
    spec = G.config_c1(seed=4, P=24, level=3, height=0.31)
    cloth = spec.meshes[0]
    cloth.v = np.zeros_like(cloth.x)
    cloth.v[:, 1] = -0.02 / (steps * spec.params.subh)
    return spec


def _analytic():
    """A self-colliding cloth over a sphere collider and a triangle obstacle."""
    from ysim_b200 import _lib, generators as G
    spec = _folded(20, 1)
    x = spec.meshes[0].x
    low = x[np.argmin(x[:, 1])].astype(np.float64)
    spec.meshes.append(G.analytic_collider(_lib.COLLIDER_SPHERE, low - (0, 0.05, 0), (0.05, 0.05, 0.05)))
    return spec


SCENES = {"off": lambda: _folded(24, 0), "hash": lambda: _folded(24, 1), "bvh": lambda: _folded(24, 2),
          "drop": lambda: _drop(8), "analytic": _analytic}


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("scene", SCENES)
@pytest.mark.parametrize("steps", [1, 8, 12])  # the first, one inside a frame, one in the next
def test_detect(cuda_lib, scene, layout, steps):
    a, b = _pair(SCENES[scene](), layout, steps)
    try:
        rows = []
        for s in (a, b):
            s.broad_phase.detect_collisions()
            rows.append(canon_rows_full(s.rows()))
            s.narrow_phase.narrow_and_sort_by_vertices()
        assert np.array_equal(rows[0], rows[1])
        assert len(rows[0]) > 0 or scene == "off" or (scene, steps) == ("drop", 1)
        (ao, ac), (bo, bc) = a.contacts(), b.contacts()
        assert np.array_equal(ao, bo) and np.array_equal(ac, bc)
        for s in (a, b):
            s.system.snapshot_xprev()
            s.system.update()
        for w in ("x", "v", "xprev"):
            assert np.array_equal(a.get(w), b.get(w))
        assert a.stats() == b.stats()
    finally:
        a.close()
        b.close()


def _slots(tree):
    """(face or -1, box) of every child slot in use, in an order of their own (node numbers are dealt by atomics)."""
    used = tree["child"] != W4_EMPTY
    box = np.concatenate([np.moveaxis(tree["lo"], 1, 2), np.moveaxis(tree["hi"], 1, 2)], 2)[used]
    child = tree["child"][used]
    t = np.column_stack([np.where(child < 0, ~child, -1).astype(np.int64), box.view(np.uint32).astype(np.int64)])
    return t[np.lexsort(t.T)]


@pytest.mark.parametrize("scene", ["hash", "bvh"])
@pytest.mark.parametrize("call", ["none", "update", "set", "set_again", "tune_set", "rebuild", "tree"])
def test_trees_outlive_their_buffers(cuda_lib, scene, call):
    """Calls between the fused substep and the reading of its trees that write its buffers or rebuild some trees; the
    obstacle moves and is not rebuilt."""
    from ysim_b200 import _lib
    spec = SCENES[scene]()
    spec.meshes[1].flags = _lib.MESH_COLLIDABLE
    spec.meshes[1].v = np.full_like(spec.meshes[1].x, 0.1)
    if call == "rebuild":
        spec.params.rebuild_frames = 1
    a, b = _pair(spec, "cube", spec.params.substeps)
    try:
        if call == "tune_set":  # the tuner refits at the current state
            a.autotune(reps=1)
            b.broad_phase.refit_swept()
        for s in (a, b):
            if call == "update":
                s.system.update()
            elif "set" in call:
                for w in ("v", "xprev", "x") * (2 if call == "set_again" else 1):
                    s.set(w, s.get(w) + np.float32(0.01))
            elif call == "rebuild":
                s.broad_phase.build()
        if call == "tree":
            assert np.array_equal(a.tree(0)[0]["mn"], b.tree(0)[0]["mn"])
        if "set" in call:
            rows = []
            for s in (a, b):
                s.broad_phase.detect_collisions()
                rows.append(canon_rows_full(s.rows()))
            assert np.array_equal(rows[0], rows[1])
        for m in range(2):
            wa, wb = _slots(a.wide_tree(m)), _slots(b.wide_tree(m))
            assert len(wa) > 0 and np.array_equal(wa, wb)
    finally:
        a.close()
        b.close()
