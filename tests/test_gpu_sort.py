"""The radix sort at the edges of its forms (one CTA, small and large tiles, groups of tiles, partial last tiles), on keys
that crowd one digit, in place, against the stable sort; the scratch's end is checked for writes past it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL, TILE, LARGE_TILE = 512 * 11, 256 * 8, 256 * 20
LARGE = 148 * LARGE_TILE


def _keys(kind, n, rng):
    if kind == "random":
        return rng.integers(0, 1 << 32, n, dtype=np.uint32)
    if kind == "equal":
        return np.full(n, 0xFFFFFFFF, np.uint32)
    if kind == "sorted":
        return np.sort(rng.integers(0, 1 << 30, n, dtype=np.uint32))[::-1].copy()
    k = rng.integers(0, 3, n, dtype=np.uint32) * np.uint32(0x01000100)  # few values, one digit constant
    k[rng.integers(0, n, max(1, n // 50))] = 0xFFFFFFFF
    return k


@pytest.mark.parametrize("kind", ["random", "equal", "sorted", "few"])
@pytest.mark.parametrize("n", [2, 31, 511, SMALL - 1, SMALL, SMALL + 1, 3 * TILE - 1, 3 * TILE, 16 * TILE, 16 * TILE + 1,
                               33 * TILE + 5, LARGE - 1, LARGE, LARGE + 1, 16 * 11 * LARGE_TILE + 1, 3_000_001])
def test_sort_edges(cuda_lib, n, kind):
    import torch
    from ysim_b200 import _lib
    rng = np.random.default_rng(n)
    keys, vals = _keys(kind, n, rng), rng.permutation(n).astype(np.uint32)
    dk, dv = (torch.from_numpy(a.view(np.int32)).cuda() for a in (keys, vals))
    size = int(cuda_lib.ys_radix_sort_scratch_bytes(n))
    for at in (0, 4):  # any 4-byte alignment was taken
        k, v = dk.clone(), dv.clone()
        buf = torch.full((size + 68,), 0x5A, dtype=torch.uint8, device="cuda")
        _lib.check(cuda_lib.ys_radix_sort_pairs(C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()), n,
                                                C.c_void_p(buf.data_ptr() + at), None))
        o = np.argsort(keys, kind="stable")
        assert np.array_equal(k.cpu().numpy().view(np.uint32), keys[o])
        assert np.array_equal(v.cpu().numpy().view(np.uint32), vals[o])
        assert bool((buf[at + size:] == 0x5A).all())
