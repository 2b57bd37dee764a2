"""The spatial hash's build at the edges of its table and sort (one sorting pass to three, an odd or even number, the
sort in one CTA, a table halved because its last bit would be a pass), of its runs (within a warp, across warps, past the
saturating length) and of its cell ordinals (boxes of up to 4096 cells, longer ones), against all pairs on the host."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs(lib, x, f, q, cell, margin, entries):
    import torch
    from ysim_b200 import _lib
    d = [torch.from_numpy(a).cuda() for a in (x, f.astype(np.int32), q)]
    p = lambda t: C.c_void_p(t.data_ptr())
    cap = 1 << 20
    out = torch.empty(cap, 2, dtype=torch.int32, device="cuda")
    n = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    h = C.c_void_p()
    _lib.check(lib.ys_shash_create(C.byref(h), len(f), entries, 0, None))
    try:
        _lib.check(lib.ys_shash_build(h, p(d[0]), p(d[1]), len(f), np.float32(cell)))
        _lib.check(lib.ys_shash_query(h, p(d[2]), len(q), np.float32(margin), p(out), cap, p(n)))
        ne, big = C.c_uint32(), C.c_uint32()
        _lib.check(lib.ys_shash_entries(h, C.byref(ne), C.byref(big)))
    finally:
        _lib.check(lib.ys_shash_destroy(h))
    n = int(n.item())
    assert n <= cap
    a = out[:n].cpu().numpy().astype(np.int64)
    return np.sort(a[:, 0] << 32 | a[:, 1]), ne.value, big.value


def _check(lib, lo, hi, cell, margin, nQ=400, seed=1):
    """Triangles with the boxes [lo, hi] (corners lo, hi and a mix of both)."""
    nF = len(lo)
    x = np.stack([lo, hi, np.where(np.arange(3) % 2, lo, hi)], 1).astype(np.float32).reshape(-1, 3)
    f = np.arange(3 * nF, dtype=np.uint32).reshape(nF, 3)
    rng = np.random.default_rng(seed)
    q = (lo[rng.integers(0, nF, nQ)] + rng.normal(0, margin, (nQ, 3))).astype(np.float32)
    m = np.float32(margin)
    a, b = q - m, q + m
    mn, mx = x.reshape(nF, 3, 3).min(1), x.reshape(nF, 3, 3).max(1)
    want = []
    for i in range(nQ):
        t = np.nonzero(((b[i] >= mn) & (a[i] <= mx)).all(1))[0]
        want.append((i << 32) | t)
    got, ne, big = _pairs(lib, x, f, q, cell, margin, 64 * 4096 + 64 * nF)
    assert np.array_equal(got, np.sort(np.concatenate(want)))
    return ne, big


# one entry a triangle: table bits 1, 5, 8, 9 -> 8, 13, 13 (above the one-CTA sort), 16, 17 -> 16, 18
@pytest.mark.parametrize("nF", [1, 16, 128, 129, 256, 5632, 5633, 32768, 32769, 65536, 65537])
def test_tables(cuda_lib, nF):
    rng = np.random.default_rng(nF)
    cell = 1.0 / 64
    lo = ((np.floor(rng.uniform(0, 64, (nF, 3))) + 0.25) * cell).astype(np.float32)
    ne, big = _check(cuda_lib, lo, (lo + np.float32(0.25 * cell)).astype(np.float32), cell, 0.4 * cell)
    assert (ne, big) == (nF, 0)


# triangles in one cell, after a few elsewhere so that the run starts anywhere in its warp
@pytest.mark.parametrize("before", [0, 1, 17, 31])
@pytest.mark.parametrize("run", [1, 14, 15, 16, 31, 32, 33, 65])
def test_runs(cuda_lib, run, before):
    cell = 1.0 / 8
    at = np.concatenate([np.stack([np.zeros(before), np.zeros(before), np.arange(before) % 4], 1), np.full((run, 3), 5.0),
                         np.full((3, 3), 6.0)])
    lo = ((at + 0.25) * cell).astype(np.float32)
    _check(cuda_lib, lo, (lo + np.float32(0.5 * cell)).astype(np.float32), cell, 0.3 * cell)


@pytest.mark.parametrize("span", [(1, 1, 1), (4096, 1, 1), (1, 4096, 1), (1, 1, 4096), (16, 16, 16), (64, 64, 1), (3, 5, 7),
                                  (1365, 3, 1), (7, 585, 1), (4097, 1, 1), (17, 16, 16)])
def test_spans(cuda_lib, span):
    cell = 1.0 / 16
    lo = np.float32([[0.3 * cell] * 3, [2.3 * cell] * 3, [0.3 * cell] * 3])
    hi = (lo + (np.float32(span) - 1) * np.float32(cell) + np.float32(0.2 * cell)).astype(np.float32)
    ne, big = _check(cuda_lib, lo, hi, cell, 0.4 * cell)
    cells = int(np.prod(span))
    assert (ne, big) == ((3 * cells, 0) if cells <= 4096 else (0, 3))
