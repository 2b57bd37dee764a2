"""Rollout passes enqueued (the first and, where substeps have branches, the first four), captured and replayed give the same bits as
passes without graphs: cloths on either side of the one-kernel limit, and the reference's trees."""
import pytest

from tests.test_gpu_adjoint_passes import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,layout", [(24, None), (200, None), (24, 0)], ids=["one_kernel", "apart", "reference"])
def test_passes(cuda_lib, N, layout):
    import torch
    from ysim_b200.adjoint import ClothRollout
    spec, k, L, v0, seed = _problem(N, 5)
    g = torch.from_numpy(seed).cuda()

    def passes(graphs):
        roll = ClothRollout(spec, 7, 3, tree_layout=layout)
        roll.scene.set_graphs(graphs)
        out = []
        for scale in (1.0, 0.8, 1.1, 0.9, 1.2, 1.0):
            p = [torch.from_numpy(a).cuda().requires_grad_() for a in (k * scale, L, v0)]
            x = roll(*p)
            out.append([x.detach().clone(), *(t.clone() for t in torch.autograd.grad(x, p, g))])
            roll.scene.step(2)
        roll.close()
        return out

    a, b = passes(True), passes(False)
    assert all(torch.equal(x, y) for s, t in zip(a, b) for x, y in zip(s, t))
    assert all(torch.equal(x, y) for x, y in zip(a[0], a[5])) and not torch.equal(a[0][0], a[1][0])
