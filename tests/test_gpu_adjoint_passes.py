"""The rollout's passes as graphs and its per-spring forms: repeated calls with new parameters, odd step counts, segments
that do not divide, scenes stepped in between, and graphs switched off give the same bits; the binary64 forms on either
side of their size rule equal the FP64 reference."""
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


@pytest.mark.parametrize("steps,every", [(1, 1), (7, 3), (12, 5), (25, 20)])
def test_float32_passes(cuda_lib, steps, every):
    import torch
    from ysim_b200.adjoint import ClothRollout
    spec, k, L, v0, seed = _problem(24, steps)
    g = torch.from_numpy(seed).cuda()

    def passes(graphs):
        roll = ClothRollout(spec, steps, every)
        roll.scene.set_graphs(graphs)
        out = []
        for scale in (1.0, 0.8, 1.0):
            p = [torch.from_numpy(a).cuda().requires_grad_() for a in ((k * np.float32(scale)), L, v0)]
            x = roll(*p)
            out += [x.detach().clone()] + [t.clone() for t in torch.autograd.grad(x, p, g)]
            out.append(torch.from_numpy(roll.scene.get("x")))
            roll.scene.step(3)  # leaves the buffers in another rotation
        out.append(torch.tensor(roll.scene.stats()["substeps"]))
        roll.close()
        return out

    a, b = passes(True), passes(False)
    assert all(torch.equal(x.cpu(), y.cpu()) for x, y in zip(a, b))
    assert torch.equal(a[0], a[10]) and not torch.equal(a[0], a[5])  # the first parameters again


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
