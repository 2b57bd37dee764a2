"""Staged calls after a fused substep: they read the trees, root boxes and grid extents of that substep's refit, as they
do after a staged substep (the two paths leave the same state, so every comparison is exact)."""
import numpy as np
import pytest

from tests.helpers import canon_rows_full
from tests.test_gpu_groups import _folded

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
    from ysim_b200 import generators as G
    spec = _folded(20, 1)
    low = float(spec.meshes[0].x[:, 1].min())
    spec.meshes.append(G.analytic_mesh(G.SPHERE, (0.1, low - 0.05, 0.0), (0.05, 0.05, 0.05)))
    return spec


SCENES = {"off": lambda: _folded(24, 0), "hash": lambda: _folded(24, 1), "bvh": lambda: _folded(24, 2),
          "drop": lambda: _drop(8), "analytic": _analytic}


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("scene", SCENES)
@pytest.mark.parametrize("steps", [1, 8, 12])  # the first, one in a frame, one after a rebuild
def test_detect(cuda_lib, scene, layout, steps):
    a, b = _pair(SCENES[scene](), layout, steps)
    try:
        rows = []
        for s in (a, b):
            s.broad_phase.detect_collisions()
            rows.append(canon_rows_full(s.rows()))
            s.narrow_phase.narrow_and_sort_by_vertices()
        assert np.array_equal(rows[0], rows[1])
        assert len(rows[0]) > 0 or (scene, steps) in (("drop", 1), ("off", 1))
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


@pytest.mark.parametrize("scene", ["hash", "bvh"])
@pytest.mark.parametrize("call", ["update", "set", "rebuild", "tree", "narrow"])
def test_trees_outlive_their_buffers(cuda_lib, scene, call):
    """Calls between the fused substep and the reading of its trees that write its buffers or rebuild some trees."""
    a, b = _pair(SCENES[scene](), "cube", 10)  # a whole frame: the next preamble may rebuild
    try:
        for s in (a, b):
            s.narrow_phase.narrow_and_sort_by_vertices()  # the contacts that update() answers, from no rows or b's
        if call == "update":
            for s in (a, b):
                s.system.update()
        elif call == "set":
            for w in ("v", "xprev", "x"):
                for s in (a, b):
                    s.set(w, s.get(w) + np.float32(0.25))
        elif call == "rebuild":
            for s in (a, b):
                s.broad_phase.build()
        elif call == "tree":
            assert all(np.array_equal(p, q) for p, q in zip(a.tree(0), b.tree(0)))
        for m in range(2):
            wa, wb = a.wide_tree(m), b.wide_tree(m)
            assert len(wa) > 0 and np.array_equal(wa, wb)
    finally:
        a.close()
        b.close()
