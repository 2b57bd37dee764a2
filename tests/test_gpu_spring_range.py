"""Spring forces over the range of lengths on either side of the bounds of the branch-free unit vector (2^-30 and 2^30 for
the length, 2^-80 for a component, a length whose significand is all ones) against the oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ONES = float(np.uint32(0x3FFFFFFF).view(np.float32))  # the float below 2


# spacing, height of the off-plane jitter relative to it
@pytest.mark.parametrize("spacing,jitter", [
    (2.0**-31, 0.3), (2.0**-29, 0.3), (1e-7, 0.3), (1e-3, 0.0), (1e-3, 1e-25), (1e-3, 2e-22), (1e-3, 0.3), (ONES, 0.0),
    (500.0, 0.3), (2.0**29, 0.3), (2.0**31, 0.3), (1e20, 0.3)])
@pytest.mark.parametrize("kind", ["grid", "triangles"])
def test_spring_lengths(cuda_lib, oracle, kind, spacing, jitter):
    from ysim_b200 import generators as G
    from ysim_b200.scene import Scene
    P = 19
    spec = G.config_c1(P=P, level=1, height=0.3) if kind == "grid" else G.config_c2(P=P, level=1, self_mode=0)
    cloth = spec.meshes[0]
    spec.meshes = [cloth]
    rng = np.random.default_rng(5)
    r, c = np.divmod(np.arange(P * P), P)
    x = np.stack([c * spacing, jitter * spacing * rng.uniform(-1, 1, P * P), r * spacing], 1).astype(np.float32)
    x[::7, 1] = -0.0
    cloth.x = x
    cloth.v = rng.normal(0, 0.1, x.shape).astype(np.float32)
    ref, gpu = oracle.OracleScene(spec), Scene(spec)
    try:
        for _ in range(2):
            ref.step(1)
            gpu.step(1)
            for w in ("x", "v"):
                a, b = gpu.get(w), ref.get(w)
                nan = np.isnan(b)
                assert np.array_equal(np.isnan(a), nan)
                assert np.array_equal(a.view(np.uint32)[~nan], b.view(np.uint32)[~nan]), w
    finally:
        gpu.close()
