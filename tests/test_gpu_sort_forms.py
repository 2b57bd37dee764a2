"""The radix sort's rarer forms: 64-bit look-back words (2^28 pairs and more), and tiles that count their predecessors' keys
themselves because those have not published their counts."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_wide_words(cuda_lib):
    import torch
    from ysim_b200 import _lib
    n = (1 << 28) + 3
    g = torch.Generator(device="cuda").manual_seed(7)
    keys = torch.randint(-2**31, 2**31, (n,), dtype=torch.int32, device="cuda", generator=g)
    keys[::3] &= 0xFF00  # long runs of equal keys
    k, v = keys.clone(), torch.arange(n, dtype=torch.int32, device="cuda")
    size = int(cuda_lib.ys_radix_sort_scratch_bytes(n))
    buf = torch.empty(size, dtype=torch.uint8, device="cuda")
    _lib.check(cuda_lib.ys_radix_sort_pairs(C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()), n,
                                            C.c_void_p(buf.data_ptr()), None))
    torch.cuda.synchronize()
    # (key, index) strictly ascending with in-range indices that carry their keys: the stable order, and only it
    for i in range(0, n, 1 << 26):
        a, b = k[i:i + (1 << 26) + 1], v[i:i + (1 << 26) + 1].long()
        assert bool(((b >= 0) & (b < n)).all()) and torch.equal(keys[b], a)
        u = a.long() & 0xFFFFFFFF
        assert bool(((u[:-1] < u[1:]) | ((u[:-1] == u[1:]) & (b[:-1] < b[1:]))).all())


@pytest.fixture(scope="module")
def counting(cuda_lib, tmp_path_factory):
    from tests import cuda_build
    lib = cuda_build.load("sort_polls", tmp_path_factory.mktemp("sort"))
    lib.sort_pairs.argtypes = [C.c_void_p, C.c_void_p, C.c_uint32]
    return lib


@pytest.mark.parametrize("n", [5633, 70_001, 757_760, 900_001])  # small tiles, several groups of them, large tiles
@pytest.mark.parametrize("top", [1 << 32, 3], ids=["random", "few"])
def test_counting(counting, n, top):
    import torch
    rng = np.random.default_rng(n)
    keys, vals = rng.integers(0, top, n, dtype=np.uint32), rng.permutation(n).astype(np.uint32)
    k, v = (torch.from_numpy(a.view(np.int32)).cuda() for a in (keys, vals))
    assert counting.sort_pairs(k.data_ptr(), v.data_ptr(), n) == 0
    o = np.argsort(keys, kind="stable")
    assert np.array_equal(k.cpu().numpy().view(np.uint32), keys[o])
    assert np.array_equal(v.cpu().numpy().view(np.uint32), vals[o])
