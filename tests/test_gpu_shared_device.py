"""Scenes stepped in turn on one GPU take more vertices per warp than one alone; their states are the same, through the
change (the fourth call in a row beside the others) and back."""
import threading

import numpy as np
import pytest

from tests.test_gpu_groups import _folded

pytestmark = pytest.mark.gpu


def _specs():
    from ysim_b200 import generators as G
    grids = G.split_instances(G.config_c4(instances=6, lo=40, hi=160, level=2, drop=0.001))
    return grids + [_folded(40, 1), _folded(60, 2)]


def _state(s):
    st = s.stats()
    return [s.get(w).view(np.uint32) for w in ("x", "v")] + [s.totals(), st["broad_rows"], st["contacts"], st["flags"]]


def _same(a, b):
    assert all(np.array_equal(p, q) for p, q in zip(a[:2], b[:2])) and a[2:] == b[2:]


@pytest.mark.parametrize("n", [1, 10], ids=["substeps", "frames"])
@pytest.mark.parametrize("threads", [False, True], ids=["one_thread", "threads"])
def test_states(cuda_lib, n, threads):
    from ysim_b200.scene import Scene
    specs, calls = _specs(), 12
    alone = []
    for spec in specs:
        s = Scene(spec)
        try:
            for _ in range(2 * calls):
                s.step(n)
            alone.append(_state(s))
        finally:
            s.close()
    scenes = [Scene(spec) for spec in specs]
    try:
        if threads:
            def run(s):
                for _ in range(calls):
                    s.step(n)
            ts = [threading.Thread(target=run, args=(s,)) for s in scenes]
            for t in ts:
                t.start()
            for t in ts:
                t.join()
        else:
            for _ in range(calls):
                for s in scenes:
                    s.step(n)
        for s in scenes:
            s.sync()
        for s in scenes:  # and each by itself again
            for _ in range(calls):
                s.step(n)
            s.sync()
        for s, a in zip(scenes, alone):
            _same(_state(s), a)
    finally:
        for s in scenes:
            s.close()
