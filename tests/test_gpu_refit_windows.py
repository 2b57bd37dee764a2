"""Boxes of the standalone tree's nodes inside one block of 256 sorted leaves, for ranges of every length up to it and trees
that end anywhere in a block: each is the union of its leaves' boxes, bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("consistent", [1, 0])
@pytest.mark.parametrize("n", [1, 2, 3, 16, 17, 64, 65, 128, 129, 255, 256, 257, 300, 511, 512, 513, 4097])
def test_ranges(cuda_lib, n, consistent):
    import torch
    from ysim_b200 import _lib
    rng = np.random.default_rng(n)
    # distinct points on a line whose gaps grow: a chain of ranges of all lengths; every other size uniform points
    t = np.cumsum(1.03 ** np.minimum(np.arange(n), 400)) if n % 2 else rng.permutation(n) + 1.0
    c = np.stack([t, rng.uniform(0, t.max() * 1e-3, n), rng.uniform(0, t.max() * 1e-3, n)], 1) / t.max()
    x = (c[:, None, :] + rng.normal(0, 1e-4, (n, 3, 3))).astype(np.float32).reshape(-1, 3)
    f = np.arange(3 * n, dtype=np.int32)
    dx, df = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
    torch.cuda.synchronize()
    h = C.c_void_p()
    _lib.check(cuda_lib.ys_lbvh_create(C.byref(h), n, 0, None))
    try:
        _lib.check(cuda_lib.ys_lbvh_set_split(h, consistent))
        _lib.check(cuda_lib.ys_lbvh_build(h, C.c_void_p(dx.data_ptr()), 3 * n, C.c_void_p(df.data_ptr()), n))
        nodes, parent, codes, idx, num = C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_uint32()
        _lib.check(cuda_lib.ys_lbvh_arrays(h, C.byref(nodes), C.byref(parent), C.byref(codes), C.byref(idx), C.byref(num)))

        class _Words:
            __cuda_array_interface__ = {"shape": (2 * n - 1, 8), "typestr": "<f4", "data": (nodes.value, False), "version": 3}
        N = torch.as_tensor(_Words(), device="cuda").cpu().numpy()
    finally:
        _lib.check(cuda_lib.ys_lbvh_destroy(h))
    ab = N.view(np.int32)[:, [3, 7]]
    box = x.reshape(n, 3, 3)
    lo, hi = box.min(1), box.max(1)
    seen = 0
    todo = [(0, False)]
    mn, mx = {}, {}
    while todo:
        i, done = todo.pop()
        a, b = ab[i]
        if a < 0:
            mn[i], mx[i] = lo[b], hi[b]
        elif not done:
            todo += [(i, True), (a, False), (b, False)]
            continue
        else:
            mn[i], mx[i] = np.minimum(mn[a], mn[b]), np.maximum(mx[a], mx[b])
        seen += 1
        assert np.array_equal(N[i, :3], mn[i]) and np.array_equal(N[i, 4:7], mx[i]), (i, a, b)
    assert seen >= (2 * n - 1 if consistent else 1)
