"""The standalone tree with the reference's midpoint split, whose boxes are range unions over the leaves each run of equal
Morton codes reaches: the oracle's boxes on every node the root reaches (built and refit), for runs of every length around the limits of
the run walk, a run across leaf blocks, runs at the ends, one run alone, and NaN corners (the climb's boxes)."""
import ctypes as C

import numpy as np
import pytest

from helpers import canon_pairs, reachable
from test_gpu_parity import _dev, _lbvh, _p, _query_pairs, _tree_equal, tree_arrays

pytestmark = pytest.mark.gpu


def _soup(runs, singles, seed):
    """Clusters of `runs` triangles, each cluster inside one Morton cell, and scattered triangles, in random order."""
    rng = np.random.default_rng(seed)
    c = [np.repeat(rng.uniform(0.05, 0.95, (1, 3)), r, axis=0) for r in runs] + [rng.uniform(0, 1, (singles, 3))]
    c = np.concatenate(c)
    tri = c[:, None, :] + rng.normal(0, 1e-6, (len(c), 3, 3))
    tri[-1] = 0.0  # the corners of the box
    tri[-2] = 1.0
    tri = tri[rng.permutation(len(tri))]
    x = tri.reshape(-1, 3).astype(np.float32)
    return x, np.arange(len(x), dtype=np.uint32).reshape(-1, 3)


CASES = {"pairs": ([2] * 50, 400), "threes": ([3] * 90, 30), "mixed": (list(range(2, 65)), 700), "limit": ([63, 64, 64], 300),
         "past_limit": ([65, 3, 2], 300), "across_blocks": ([64] * 9, 2), "one_run": ([40], 2), "many": ([3, 4, 5, 7] * 900, 20000)}


@pytest.mark.parametrize("case", CASES)
def test_boxes_are_the_reference_trees(cuda_lib, oracle, case):
    from ysim_b200 import _lib
    x, f = _soup(*CASES[case], seed=len(case))
    v = np.random.default_rng(1).normal(0, 1e-2, x.shape).astype(np.float32)
    onodes = oracle.build_tree(x, f)[0]
    h, dx, df = _lbvh(cuda_lib, x, f)
    try:
        nodes = tree_arrays(cuda_lib, h)[0]
        _tree_equal(nodes, onodes)
        q = (x[::7] + np.float32(1e-4)).astype(np.float32)
        dv = _dev(v.reshape(-1))
        for _ in range(2):
            _lib.check(cuda_lib.ys_lbvh_refit(h, _p(dx), _p(dv), np.float32(1e-2), 1))
            onodes = oracle.refit(onodes, x, v, f, np.float32(1e-2), True)
            nodes = tree_arrays(cuda_lib, h)[0]
            _tree_equal(nodes, onodes)
        want = canon_pairs(oracle.query_points(onodes, f, q, 1e-3))
        assert np.array_equal(_query_pairs(cuda_lib, h, q, np.float32(1e-3)), want)
    finally:
        _lib.check(cuda_lib.ys_lbvh_destroy(h))


def test_nan_corner(cuda_lib, oracle):
    """A refit that meets NaN gives the climb's boxes, and the next one without it the range unions again."""
    from ysim_b200 import _lib
    x, f = _soup([3] * 20, 300, 5)
    bad = x.copy()
    bad[17, 1] = np.nan
    onodes = oracle.build_tree(x, f)[0]
    h, dx, df = _lbvh(cuda_lib, x, f)
    try:
        for a in (bad, x, bad, x):
            _lib.check(cuda_lib.ys_lbvh_refit(h, _p(_dev(a.reshape(-1))), None, np.float32(0), 0))
            onodes = oracle.refit(onodes, a, x, f, np.float32(0), False)
            nodes = tree_arrays(cuda_lib, h)[0]
            r = reachable(onodes)  # as _tree_equal, with NaN equal to NaN
            for k in ("mn", "mx"):
                assert np.array_equal(nodes[k][r], onodes[k][r], equal_nan=True)
    finally:
        _lib.check(cuda_lib.ys_lbvh_destroy(h))
