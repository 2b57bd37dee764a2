"""The fused substep's descent over sorted-leaf groups at the edges of its runs of 32, 1024 and 32768 leaves, and the
box sets a mesh can need, against the oracle (bit for bit, as the substep's arithmetic is the oracle's)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _folded(P, self_mode, seed=3):
    """A P x P cloth folded in two, half a spacing between its closing layers, over a small obstacle; (spec, v)."""
    from ysim_b200 import generators as G
    spec = G.config_c2(seed=seed, P=P, level=2, self_mode=self_mode, gravity=-9.81)
    spec.params.cols_per_point = 60  # room for every row in the oracle (the fused path stores none)
    cloth, obst = spec.meshes
    s = 1.0 / (P - 1)
    x = cloth.x - np.float32([0, 0.37, 0])
    up = x[:, 0] >= 0
    x = np.stack([np.abs(x[:, 0]) - 0.25, x[:, 1] + np.where(up, 0.25, -0.25) * s, x[:, 2]], 1)
    x[:, 1] += float(obst.x[:, 1].max()) + 0.3 * s - x[:, 1].min()
    cloth.x = x.astype(np.float32)
    cloth.v = np.zeros_like(cloth.x)
    cloth.v[up, 1] = -60 * s
    return spec


def _against_oracle(oracle, spec, steps=3):
    from ysim_b200.scene import Scene
    ref, gpu = oracle.OracleScene(spec), Scene(spec)
    try:
        gpu.set_record(True)
        rows = 0
        for _ in range(steps):
            ref.step(1)
            gpu.step(1)
            for w in ("x", "v"):
                assert np.array_equal(gpu.get(w).view(np.uint32), ref.get(w).view(np.uint32)), w
            goff, gc = gpu.contacts()
            roff, rc = ref.contacts()
            assert np.array_equal(goff, roff)
            for k in ("tobj", "tri"):
                assert np.array_equal(gc[k], rc[k])
            g, r = gpu.stats(), ref.stats()
            assert g["broad_rows"] == r["broad_rows"] and g["flags"] == r["flags"] == 0
            rows += g["broad_rows"]
        return rows
    finally:
        gpu.close()


# faces: 2, 8, 32, 50, 968, 1058, 2048, 32768, 33282
@pytest.mark.parametrize("self_mode", [1, 2], ids=["hash", "bvh"])
@pytest.mark.parametrize("P", [2, 3, 5, 6, 23, 24, 33, 129, 130])
def test_runs_of_leaves(cuda_lib, oracle, P, self_mode):
    assert _against_oracle(oracle, _folded(P, self_mode)) > 0 or P < 6


@pytest.mark.parametrize("self_mode", [0, 1, 2], ids=["off", "hash", "bvh"])
def test_box_sets(cuda_lib, oracle, self_mode):
    """Self-colliding cloths that are each other's targets (key and query boxes of one mesh), a vertex on no face (root
    box by faces), a moving obstacle, cloths small enough to share a warp and, with hash rows, a cloth marked static (its
    faces are refit for the grid extent; under the other modes a static mesh's faces stay as they were built, also when
    it is a cloth and moves)."""
    from ysim_b200 import _lib, generators as G
    spec = _folded(20, self_mode)
    cloth, obst = spec.meshes
    s = 1.0 / 19
    other = dataclasses.replace(cloth, x=(cloth.x + np.float32([0.013, 1.2 * s, 0.007])).astype(np.float32))
    loose = dataclasses.replace(  # one more vertex, on no face
        cloth, x=np.concatenate([cloth.x + np.float32([0, 2.4 * s, 0]), np.float32([[0.1, 2.0, 0.1]])]),
        v=np.concatenate([cloth.v, np.zeros((1, 3), np.float32)]), mass=np.full(401, 1e-2, np.float32),
        mask=np.ones(401, np.float32))
    below = dataclasses.replace(cloth, x=(cloth.x - np.float32([0, 0.9 * s, 0])).astype(np.float32),
                                v=np.zeros_like(cloth.v), flags=cloth.flags | (_lib.MESH_STATIC if self_mode == 1 else 0))
    moving = dataclasses.replace(obst, flags=_lib.MESH_COLLIDABLE, behavior=_lib.KINEMATIC,
                                 v=np.full_like(obst.x, 0.1))
    tiny = []
    for k in range(5):
        x, f = G.grid_cloth(3, 0.05, (0.06 * k, float(other.x[:, 1].max()) + 0.2 * s, 0.1))
        tiny.append(G.Mesh(behavior=_lib.TRIANGULAR_CLOTH, flags=cloth.flags, x=x, facets=f, v=np.zeros_like(x),
                           mass=np.full(9, 1e-2, np.float32), mask=np.ones(9, np.float32), kstretch=1e3, kbend=10.0,
                           thickness=cloth.thickness))
    spec.meshes = [cloth, *tiny[:2], other, loose, below, moving, *tiny[2:]]
    assert _against_oracle(oracle, spec, steps=4) > 0


# the last count of vertices with 2, 4, 8 and 16 per warp, and one more
@pytest.mark.parametrize("n", [9472, 9473, 18944, 18945, 75776, 75777, 151552, 151553])
def test_vertices_per_warp(cuda_lib, oracle, n):
    """The same states whatever the warps' share: a self-colliding cloth filled up with loose vertices to n."""
    spec = _folded(60, 1)
    cloth = spec.meshes[0]
    k = n - cloth.nV
    loose = np.random.default_rng(n).uniform(-0.3, 0.3, (k, 3)).astype(np.float32) + np.float32([0, 0.3, 0])
    spec.meshes[0] = dataclasses.replace(
        cloth, x=np.concatenate([cloth.x, loose]), v=np.concatenate([cloth.v, np.zeros_like(loose)]),
        mass=np.full(n, 1e-2, np.float32), mask=np.ones(n, np.float32))
    assert _against_oracle(oracle, spec, steps=2) > 0
