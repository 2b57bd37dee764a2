"""Whole frames enqueued or replayed as one graph: any mix of single substeps and frames, across rebuilds, state resets, a
switch of the graphs and reads in between gives the same bits as single substeps without graphs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spec(kind):
    from ysim_b200 import generators as G
    spec = G.config_c2(P=24, level=2, self_mode=1) if kind == "self" else G.config_c4(instances=3, lo=9, hi=40, level=2, drop=0.001)
    spec.params.rebuild_frames = 3
    return spec


# substeps per frame: none as a graph (1), odd, the default, the longest frame that is one graph, longer
@pytest.mark.parametrize("substeps", [1, 7, 20, 32, 33])
@pytest.mark.parametrize("kind,layout", [("self", "cube"), ("batch", "cube"), ("self", "reference")])
def test_frames(cuda_lib, kind, layout, substeps):
    from ysim_b200 import _lib
    from ysim_b200.scene import Scene
    spec = _spec(kind)
    spec.params.substeps = substeps
    f = substeps
    # whole frames until every rotation state has its graph, then ragged counts, a reset and frames again
    moves = [f] * 52 + [3 * f, 2 * f + 1, f, 2 * f - 1, "read", f, "reset", 11 * f, "graphs", f, "graphs", 2 * f, 1, 1, f]
    out = []
    for graphs in (True, False):
        s = Scene(spec, tree_layout=_lib.TREE_REFERENCE if layout == "reference" else None)
        try:
            s.set_graphs(graphs)
            on, seen = graphs, []
            start = {w: s.get(w) for w in ("x", "xprev", "v")}
            for m in moves:
                if m == "read":
                    seen += [s.get("x"), s.get("v")]
                elif m == "reset":
                    for w, a in start.items():
                        s.set(w, a)
                elif m == "graphs":
                    on = graphs and not on
                    s.set_graphs(on)
                else:
                    for _ in range(1 if graphs else m):  # single substeps where the graphs are off
                        s.step(m if graphs else 1)
            st = s.stats()
            out.append((seen + [s.get("x"), s.get("v")], s.totals(), st["broad_rows"], st["contacts"], st["flags"]))
        finally:
            s.close()
    a, b = out
    for p, q in zip(a[0], b[0]):
        assert np.array_equal(p.view(np.uint32), q.view(np.uint32))
    assert a[1:] == b[1:]
