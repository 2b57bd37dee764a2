"""A packed scene has its trees, levels and thread order before its first substep: both autotuners on a scene that has not
stepped, and a scene that never rebuilds (its first frame is that of one that does), against the oracle bit for bit."""
import numpy as np
import pytest

from tests.test_gpu_groups import _folded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", ["no_rebuilds", "autotune", "autotune_classes"])
@pytest.mark.parametrize("self_mode", [0, 1, 2], ids=["off", "hash", "bvh"])
def test_first_frame(cuda_lib, oracle, self_mode, first):
    from ysim_b200.scene import Scene
    spec = _folded(20, self_mode)
    ref = oracle.OracleScene(_folded(20, self_mode))
    if first == "no_rebuilds":
        spec.params.rebuild_frames = 0
    gpu = Scene(spec)
    try:
        if first != "no_rebuilds":
            getattr(gpu, first)(reps=2)
            gpu.broad_phase.detect_collisions()  # reads the trees that the tuner left
        for _ in range(3):
            ref.step(1)
            gpu.step(1)
            for w in ("x", "v"):
                assert np.array_equal(gpu.get(w).view(np.uint32), ref.get(w).view(np.uint32))
            assert gpu.stats()["broad_rows"] == ref.stats()["broad_rows"] and gpu.stats()["flags"] == 0
    finally:
        gpu.close()
