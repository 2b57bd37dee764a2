"""The binary64 rollout's contacts are those of a search over all faces, also where runs of equal Morton codes leave faces
that no path of the reference's midpoint-split tree reaches."""
import numpy as np
import pytest

from tests.test_gpu_adjoint import _f32_spec, _problem, _roll64, _small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [None, 0], ids=["cube", "reference"])
def test_all_faces(cuda_lib, layout):
    import torch
    spec = _f32_spec(_small(height=0.2995))
    obst = spec.meshes[1]
    # a triangle far off: the sphere's faces share a few cells of the codes' grid
    n = obst.nV
    obst.x = np.concatenate([obst.x, np.float32([[900, -1000, 900], [1000, -1000, 900], [900, -1000, 1000]])])
    obst.facets = np.concatenate([obst.facets, np.array([[n, n + 1, n + 2]], obst.facets.dtype)])
    obst.v = obst.mass = obst.mask = None
    k, L, v0, w, R = _problem(spec)
    w64 = w.astype(np.float64)
    x64, ncontacts = R.forward(40, keep=True)
    assert ncontacts > 0
    want = R.backward(40, w64)
    roll, p = _roll64(spec, k, L, v0, 40, K=7, tree_layout=layout)
    try:
        codes = roll.scene.tree(1)[2]
        assert np.unique(codes, return_counts=True)[1].max() > 64
        xT = roll(*p)
        assert np.array_equal(xT.detach().cpu().numpy(), x64)
        (xT * torch.tensor(w64, device="cuda")).sum().backward()
        for t, g in zip(p, want):
            assert np.array_equal(t.grad.cpu().numpy(), g)
    finally:
        roll.close()
