"""The kernel that refits the groups and evaluates the forces of small scenes, at its limit of two blocks per SM and with
every kind of block in one launch, against the oracle (bit for bit)."""
import dataclasses

import numpy as np
import pytest

from tests.test_gpu_groups import _against_oracle, _folded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [0, 1], ids=["last_in_one", "first_apart"])
def test_limit(cuda_lib, oracle, over):
    import torch
    spec = _folded(60, 1)
    cloth, obst = spec.meshes
    refit = -(-cloth.nF // 1024)
    blocks = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    n = 128 * (blocks - refit) + over - obst.nV
    loose = np.random.default_rng(n).uniform(-0.3, 0.3, (n - cloth.nV, 3)).astype(np.float32) + np.float32([0, 0.3, 0])
    spec.meshes[0] = dataclasses.replace(
        cloth, x=np.concatenate([cloth.x, loose]), v=np.concatenate([cloth.v, np.zeros_like(loose)]),
        mass=np.full(n, 1e-2, np.float32), mask=np.ones(n, np.float32))
    assert _against_oracle(oracle, spec, steps=2) > 0


@pytest.mark.parametrize("self_mode", [0, 1, 2], ids=["off", "hash", "bvh"])
@pytest.mark.parametrize("side", [8, 16, 17, 40])
def test_kinds_of_block(cuda_lib, oracle, side, self_mode):
    """A grid cloth (tiles), a triangle cloth (vertices), a moving obstacle."""
    from ysim_b200 import _lib, generators as G
    spec = _folded(20, self_mode)
    cloth, obst = spec.meshes
    grid = G.config_c1(P=side, level=1).meshes[0]
    grid.x = grid.x + np.float32([0, float(cloth.x[:, 1].max()) + 0.02 - float(grid.x[:, 1].min()), 0])
    obst.flags, obst.behavior, obst.v = _lib.MESH_COLLIDABLE, _lib.KINEMATIC, np.full_like(obst.x, 0.1)
    spec.params.subh = 1.0 / 6000.0  # the grid cloth's springs
    spec.meshes = [grid, cloth, obst]
    _against_oracle(oracle, spec, steps=4)
