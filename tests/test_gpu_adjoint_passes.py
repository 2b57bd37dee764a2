"""The binary64 rollout's forms on either side of their size rule equal the FP64 reference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(N, seed, level=2):
    from ysim_b200 import generators as G
    spec = G.config_c5(seed=seed, N=N, level=level, height=0.3009)
    m = spec.meshes[0]
    k, L = G.grid_spring_params(N, m.grid_rest, (m.kstretch, m.kshear, m.kbend))
    rng = np.random.default_rng(seed)
    k = (k * np.exp(rng.normal(0, 0.1, k.shape))).astype(np.float32)
    v0 = rng.normal((0, -0.3, 0), 0.01, m.x.shape).astype(np.float32)
    return spec, k, L, v0, rng.normal(0, 1, m.x.shape).astype(np.float32)


@pytest.mark.parametrize("N", [3, 4, 17, 256, 257])  # 257^2 vertices: a thread per vertex
def test_float64_forms(cuda_lib, oracle, N):
    import torch
    from ysim_b200.adjoint import ClothRollout
    from test_gpu_adjoint import _f32_spec
    spec, k, L, v0, seed = _problem(N, N)
    spec = _f32_spec(spec)
    ref = oracle.Rollout(spec, k, L, v0=v0)
    x64, _ = ref.forward(5, keep=True)
    grads = ref.backward(5, seed.astype(np.float64))
    roll = ClothRollout(spec, 5, 2, precision=64)
    try:
        p = [torch.tensor(np.asarray(a, np.float64), device="cuda", requires_grad=True) for a in (k, L, v0)]
        x = roll(*p)
        assert np.array_equal(x.detach().cpu().numpy(), x64)
        for got, want in zip(torch.autograd.grad(x, p, torch.from_numpy(seed).cuda().double()), grads):
            assert np.array_equal(got.cpu().numpy().reshape(-1), np.asarray(want).reshape(-1))
    finally:
        roll.close()
