"""Workloads of the cloth simulation library, one pass of each through its public entry points.

Nine kinds of work, each over the range of sizes that programs give it:

  drop      a FastGridCloth lands on a static triangle obstacle (real-time scenes)
  fold      a folded, self-colliding TriangularCloth lands on a static obstacle (garment scenes)
  drape     the same cloth 500 substeps into its drape over the obstacle (the benchmark's contact phase)
  batch     many FastGridCloth instances of mixed sizes, each over its own obstacle (sampling, training data)
  rollout   a differentiable FastGridCloth rollout, forward and backward (parameter fitting)
  bvh       a linear BVH over a triangle soup: build, swept refit, point query
  hash      the point-triangle spatial hash over the same soups: build, point query
  facehash  the face-face spatial hash over a packed scene
  sort      the radix sort of (key, value) pairs

A scene's pass is an episode: the program puts the cloth into its start state, steps a few frames and reads the
state back.  Pairs and rows come out of the queries in no particular order; the passes sort them, as a program does
that hands them on by vertex.
"""
import ctypes as C
import math

import numpy as np
import torch

from ysim_b200 import _lib
from ysim_b200 import generators as G
from ysim_b200.adjoint import ClothRollout
from ysim_b200.scene import Scene, Simulator


def listed():
    return [
        # the smallest interactive scene: 4096 vertices, latency and launches decide
        {"name": "drop_64", "kind": "drop", "side": 64, "level": 4, "frames": 20},
        # a garment-sized self-colliding cloth of odd side, hash-semantics self rows
        {"name": "fold_97", "kind": "fold", "side": 97, "level": 5, "self_mode": 1, "frames": 2},
        # the headline scene: 262,144 self-colliding vertices over 327,680 obstacle triangles, in contact
        {"name": "drape_512", "kind": "drape", "side": 512, "level": 7, "self_mode": 1, "frames": 5},
        # a batch of instances with sides from 16 to 256, over a million vertices in one scene
        {"name": "batch_48", "kind": "batch", "instances": 48, "lo": 16, "hi": 256, "mix": 4, "frames": 10},
        # fitting 97k spring parameters through a rollout into contact, binary32
        {"name": "rollout_128", "kind": "rollout", "side": 128, "steps": 100, "every": 20, "bits": 32},
        # the same in binary64 for gradients checked against finite differences, odd side
        {"name": "rollout_65_f64", "kind": "rollout", "side": 65, "steps": 100, "every": 20, "bits": 64},
        # a small collider's tree, rebuilt, refit and queried at every use
        {"name": "bvh_5k", "kind": "bvh", "triangles": 5120, "queries": 4096, "consistent": False},
        # a million triangles, every leaf reported exactly once
        {"name": "bvh_1m", "kind": "bvh", "triangles": 1000000, "queries": 1000000, "consistent": True},
        # four million triangles, the reference's tree node for node
        {"name": "bvh_4m", "kind": "bvh", "triangles": 4000000, "queries": 4000000, "consistent": False},
        # the spatial hash on the same soup as an alternative broad phase
        {"name": "hash_1m", "kind": "hash", "triangles": 1000000, "queries": 1000000},
        # face-face rows of a cloth over its obstacle
        {"name": "facehash_128", "kind": "facehash", "side": 128, "level": 5},
        # sorting keys of a few million primitives, a size off every tile
        {"name": "sort_3m", "kind": "sort", "pairs": 3000001},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["drop", "fold", "drape", "batch", "rollout", "bvh", "hash", "facehash", "sort"])
    if kind == "drop":
        return {"kind": kind, "side": rng.randint(17, 256), "level": rng.randint(2, 5), "frames": rng.randint(10, 20)}
    if kind == "fold":
        return {"kind": kind, "side": rng.randint(24, 200), "level": rng.randint(3, 6), "self_mode": rng.choice([1, 2]),
                "frames": rng.randint(1, 2)}
    if kind == "drape":
        return {"kind": kind, "side": rng.randint(320, 512), "level": rng.randint(6, 7), "self_mode": rng.choice([1, 2]),
                "frames": rng.randint(2, 5)}
    if kind == "batch":
        return {"kind": kind, "instances": rng.randint(3, 40), "lo": 16, "hi": rng.randint(48, 240),
                "mix": rng.randint(1, 1000), "frames": rng.randint(4, 10)}
    if kind == "rollout":
        return {"kind": kind, "side": rng.randint(20, 128), "steps": rng.randint(40, 100), "every": rng.choice([10, 20, 25]),
                "bits": rng.choice([32, 32, 64])}
    if kind == "bvh":
        n = _log_int(rng, 1000, 4000000)
        return {"kind": kind, "triangles": n, "queries": max(1000, int(n * rng.uniform(0.25, 1.0))),
                "consistent": rng.random() < 0.5}
    if kind == "hash":
        n = _log_int(rng, 5000, 2000000)
        return {"kind": kind, "triangles": n, "queries": max(1000, int(n * rng.uniform(0.25, 1.0)))}
    if kind == "facehash":
        return {"kind": kind, "side": rng.randint(32, 160), "level": rng.randint(3, 6)}
    return {"kind": kind, "pairs": _log_int(rng, 1000, 16000000)}


# ------------------------------------------------------------------ inputs
def _rng(seed):
    return np.random.Generator(np.random.PCG64(seed))


def _off_axis(rng, x):
    """x moved sideways by up to 0.02, so that no row of vertices lies along the obstacle's edges."""
    return (x + rng.uniform(-0.02, 0.02, 3) * (1.0, 0.0, 1.0)).astype(np.float32)


def _drop_start(rng, x, cloth, nV, subh):
    """The first `cloth` vertices of x off the obstacle's axis and moving down at about 1 m/s."""
    x[:cloth] = _off_axis(rng, x[:cloth])
    v = np.zeros((nV, 3), np.float32)
    v[:cloth] = rng.normal((0.0, -1.0, 0.0), 0.02, (cloth, 3))
    xprev = (x - v * np.float32(subh)).astype(np.float32)
    return {"x": x, "xprev": xprev, "v": v}


def _scene(case, seed):
    """(scene description, start state) of a scene kind; the drape's start state comes from stepping the scene."""
    rng = _rng(seed)
    if case["kind"] == "drop":
        # a sheet one and a half thicknesses above the obstacle's top: it lands within the episode
        spec = G.config_c1(seed=seed, P=case["side"], level=case["level"], height=0.3015)
        x = np.concatenate([m.x for m in spec.meshes])
        return spec, _drop_start(rng, x, spec.meshes[0].nV, spec.nV, spec.params.subh)
    if case["kind"] == "batch":
        spec = G.config_c4(seed=case["mix"], instances=case["instances"], lo=case["lo"], hi=case["hi"], drop=0.0015)
        x = np.concatenate([m.x for m in spec.meshes])
        v = np.zeros_like(x)
        at = 0
        for m in spec.meshes:
            if m.grid_n:
                x[at:at + m.nV, 1] += rng.uniform(0.0, 1e-4, m.nV).astype(np.float32)
                v[at:at + m.nV] = rng.normal((0.0, -1.0, 0.0), 0.02, (m.nV, 3))
            at += m.nV
        return spec, {"x": x, "xprev": (x - v * np.float32(spec.params.subh)).astype(np.float32), "v": v}
    spec = G.config_c2(seed=seed, P=case["side"], level=case["level"], self_mode=case["self_mode"])
    if case["kind"] == "drape":
        return spec, None
    # folded in two over its obstacle, the layers half a spacing apart and closing, the lower one about to land
    cloth, obst = spec.meshes
    s = 1.0 / (case["side"] - 1)
    flat = cloth.x.astype(np.float64) - (0.0, 0.37, 0.0)
    up = flat[:, 0] >= 0.0
    xc = np.stack([np.abs(flat[:, 0]) - 0.25, flat[:, 1] + np.where(up, 0.25, -0.25) * s, flat[:, 2]], 1)
    xc[:, 1] += float(obst.x[:, 1].max()) + s - xc[:, 1].min()
    v = np.zeros((spec.nV, 3), np.float32)
    v[:cloth.nV] = rng.normal(0.0, 0.02, (cloth.nV, 3)) + np.stack(
        [np.zeros(cloth.nV), np.where(up, -60.0 * s - 0.5, -0.5), np.zeros(cloth.nV)], 1)
    x = np.concatenate([xc.astype(np.float32), obst.x])
    return spec, {"x": x, "xprev": (x - v * np.float32(spec.params.subh)).astype(np.float32), "v": v}


def _rollout(case, seed):
    """(scene description, per-spring stiffness and rest length, initial velocity, target) of a rollout."""
    rng = _rng(seed)
    spec = G.config_c5(seed=seed, N=case["side"], height=0.303)
    m = spec.meshes[0]
    m.x = _off_axis(rng, m.x)
    k, L = G.grid_spring_params(case["side"], m.grid_rest, (m.kstretch, m.kshear, m.kbend))
    k = (k * np.exp(rng.normal(0.0, 0.1, k.shape))).astype(np.float32)
    v0 = rng.normal((0.0, -0.2, 0.0), 0.01, m.x.shape).astype(np.float32)
    target = (m.x + rng.normal((0.0, -0.1, 0.0), 0.02, m.x.shape)).astype(np.float32)
    return spec, k, L, v0, target


def _soup(n, nq, seed):
    """The collision microbenchmark's soup (centroids uniform in the unit cube, log-normal sizes) and query points."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    def uniform(*shape):
        return torch.rand(*shape, generator=g, device="cuda")
    sigma = torch.exp(torch.randn(n, 1, 1, generator=g, device="cuda") * 0.5 + math.log(1e-3))
    x = (uniform(n, 1, 3) + torch.randn(n, 3, 3, generator=g, device="cuda") * sigma).reshape(-1, 3).contiguous()
    v = torch.randn(3 * n, 3, generator=g, device="cuda") * 0.1
    f = torch.arange(3 * n, dtype=torch.int32, device="cuda")
    return x, v, f, uniform(nq, 3)


# ------------------------------------------------------------------ passes
def _p(t):
    return C.c_void_p(t.data_ptr())


class _Words:
    """Device memory of a handle as a torch tensor of 32-bit words (no copy; the tensor keeps the handle)."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<i4", "data": (ptr, False), "version": 3}


def _sorted_into(out, words, count):
    """The first `count` words in ascending order at the front of out, the rest of it -1."""
    n = min(int(count.item()), len(words), len(out))
    out.fill_(-1)
    out[:n] = torch.sort(words[:n]).values
    return out


def _sorted_room(case):
    """Room for a soup query's pairs: about 1e-7 of the products meet."""
    return 4096 + int(3e-7 * case["triangles"] * case["queries"])


class _Episode:
    def __init__(self, case, seed):
        spec, start = _scene(case, seed)
        self.scene = Scene(spec)
        self.simulator = Simulator(self.scene)
        self.frames = case["frames"]
        if start is None:
            self.scene.step(500)
            start = {w: self.scene.get(w) for w in ("x", "xprev", "v")}
        self.keep = {w: torch.from_numpy(a).pin_memory() for w, a in start.items()}
        self.start = {w: t.numpy() for w, t in self.keep.items()}
        self.x = torch.empty(spec.nV, 3, pin_memory=True)

    def __call__(self):
        s = self.scene
        for which, a in self.start.items():
            s.set(which, a)
        for _ in range(self.frames):
            self.simulator.update()
        _lib.check(s.lib.ys_scene_read_positions_async(s.h, _p(self.x)), "ys_scene_read_positions_async")
        v, st = s.get("v"), s.stats()
        return {"x": self.x, "v": v, "rows": st["broad_rows"], "contacts": st["contacts"], "flags": st["flags"]}


class _Fit:
    def __init__(self, case, seed):
        spec, k, L, v0, target = _rollout(case, seed)
        kind = torch.float64 if case["bits"] == 64 else torch.float32
        self.roll = ClothRollout(spec, case["steps"], case["every"], precision=case["bits"])
        self.k, self.L, self.v0 = (torch.from_numpy(a).cuda().to(kind).requires_grad_() for a in (k, L, v0))
        self.target = torch.from_numpy(target).cuda().to(kind)

    def __call__(self):
        x = self.roll(self.k, self.L, self.v0)
        loss = ((x - self.target) ** 2).sum(1).mean()
        gk, gL, gv = torch.autograd.grad(loss, (self.k, self.L, self.v0))
        return {"x": x.detach(), "gk": gk, "gL": gL, "gv": gv}


class _Handle:
    """A handle of the C interface, given back with the object."""

    def __init__(self, kind, *args):
        self.lib = _lib.load()
        self.h = C.c_void_p()
        self.kind = kind
        _lib.check(getattr(self.lib, f"ys_{kind}_create")(C.byref(self.h), *args, 0, None), f"ys_{kind}_create")

    def call(self, name, *args):
        _lib.check(getattr(self.lib, f"ys_{self.kind}_{name}")(self.h, *args), f"ys_{self.kind}_{name}")

    def __del__(self):
        getattr(self.lib, f"ys_{self.kind}_destroy")(self.h)


class _Bvh:
    def __init__(self, case, seed):
        n = case["triangles"]
        self.x, self.v, self.f, self.q = _soup(n, case["queries"], seed)
        self.pairs = torch.empty(_sorted_room(case), dtype=torch.int64, device="cuda")  # (point, triangle) a word
        self.sorted = torch.empty_like(self.pairs)
        self.count = torch.zeros(1, dtype=torch.int64, device="cuda")
        self.tree = _Handle("lbvh", n)
        self.tree.call("set_split", int(case["consistent"]))
        nodes, parent, codes, idx, num = C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_uint32()
        self.tree.call("arrays", C.byref(nodes), C.byref(parent), C.byref(codes), C.byref(idx), C.byref(num))
        def words(ptr, *shape):
            return torch.as_tensor(_Words(self.tree, ptr.value, shape), device="cuda")
        self.nodes, self.codes, self.idx = words(nodes, 2 * n - 1, 8), words(codes, n), words(idx, n)

    def __call__(self):
        n = self.f.numel() // 3
        self.tree.call("build", _p(self.x), 3 * n, _p(self.f), n)
        self.tree.call("refit", _p(self.x), _p(self.v), C.c_float(1e-3), 1)
        self.tree.call("query", _p(self.q), len(self.q), C.c_float(1e-3), 0, _p(self.pairs), self.pairs.numel(),
                       _p(self.count))
        return {"nodes": self.nodes, "codes": self.codes, "idx": self.idx,
                "pairs": _sorted_into(self.sorted, self.pairs, self.count)}


class _Hash:
    def __init__(self, case, seed):
        n = case["triangles"]
        self.x, _, self.f, self.q = _soup(n, case["queries"], seed)
        self.pairs = torch.empty(_sorted_room(case), dtype=torch.int64, device="cuda")  # (point, triangle) a word
        self.sorted = torch.empty_like(self.pairs)
        self.count = torch.zeros(1, dtype=torch.int64, device="cuda")
        self.hash = _Handle("shash", n, 40 * n)

    def __call__(self):
        self.hash.call("build", _p(self.x), _p(self.f), self.f.numel() // 3, C.c_float(2e-3))
        self.hash.call("query", _p(self.q), len(self.q), C.c_float(1e-3), _p(self.pairs), self.pairs.numel(),
                       _p(self.count))
        return _sorted_into(self.sorted, self.pairs, self.count)


class _FaceHash:
    def __init__(self, case, seed):
        spec = G.config_c2(seed=seed, P=case["side"], level=case["level"], height=0.36)
        ms = spec.meshes
        def dev(a):
            return torch.from_numpy(np.ascontiguousarray(a)).cuda()
        self.x = dev(np.concatenate([m.x for m in ms]).astype(np.float32))
        self.facets = dev(np.concatenate([m.facets for m in ms]).astype(np.int32))
        self.voff = dev(np.cumsum([0] + [m.nV for m in ms]).astype(np.int32))
        self.foff = dev(np.cumsum([0] + [m.nF for m in ms]).astype(np.int32))
        self.behavior = dev(np.array([m.behavior for m in ms], np.int32))
        self.shape = torch.zeros(len(ms), dtype=torch.int32, device="cuda")
        self.margin = spec.params.margin
        nF = len(self.facets)
        self.rows = torch.empty(72 * nF, 8, dtype=torch.int32, device="cuda")
        self.sorted = torch.empty(len(self.rows), dtype=torch.int64, device="cuda")
        self.count = torch.zeros(1, dtype=torch.int64, device="cuda")
        self.hash = _Handle("shff", nF)

    def __call__(self):
        self.hash.call("detect", _p(self.x), len(self.x), _p(self.voff), _p(self.facets), _p(self.foff),
                       len(self.facets), _p(self.behavior), _p(self.shape), len(self.shape), C.c_float(self.margin), 1,
                       _p(self.rows), len(self.rows), _p(self.count))
        # point, triangle and the two meshes of each row in one sortable word
        r = self.rows[:min(int(self.count.item()), len(self.rows)), :4].to(torch.int64)
        words = (r[:, 2] << 62) | (r[:, 3] << 60) | (r[:, 0] << 30) | r[:, 1]
        return _sorted_into(self.sorted, words, self.count)


class _Sort:
    def __init__(self, case, seed):
        n = case["pairs"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        # 30-bit Morton-like keys, as the trees' builds have them, and the primitives' numbers
        self.source = torch.randint(0, 1 << 30, (n,), generator=g, device="cuda", dtype=torch.int32)
        self.number = torch.arange(n, dtype=torch.int32, device="cuda")
        self.keys, self.vals = torch.empty_like(self.source), torch.empty_like(self.source)
        self.lib = _lib.load()
        self.scratch = torch.empty(self.lib.ys_radix_sort_scratch_bytes(n), dtype=torch.uint8, device="cuda")

    def __call__(self):
        self.keys.copy_(self.source)
        self.vals.copy_(self.number)
        _lib.check(self.lib.ys_radix_sort_pairs(_p(self.keys), _p(self.vals), self.keys.numel(), _p(self.scratch), None),
                   "ys_radix_sort_pairs")
        return {"keys": self.keys, "vals": self.vals}


_PASS = {"drop": _Episode, "fold": _Episode, "drape": _Episode, "batch": _Episode, "rollout": _Fit, "bvh": _Bvh,
         "hash": _Hash, "facehash": _FaceHash, "sort": _Sort}


def prepare(case, seed):
    return _PASS[case["kind"]](case, seed)


def run(state):
    return state()


# ------------------------------------------------------------------ work
def _grid_springs(n):
    return 2 * n * (n - 1) + 2 * (n - 1) ** 2 + 2 * n * (n - 2)


def work(case):
    """Per substep the state is read and written once (positions, previous positions, velocities, mass and mask in,
    positions and velocities out: 68 bytes a vertex) and each of the springs and triangles is read once."""
    kind = case["kind"]
    if kind in ("drop", "fold", "drape"):
        n, obstacle = case["side"], 20 * 4 ** case["level"]
        V, M = n * n, 2 * (n - 1) ** 2
        substeps = case["frames"] * (10 if kind == "drop" else 20)
        springs = 0 if kind == "drop" else 16 * (3 * M // 2)
        step = 68 * V + springs + (12 * M if kind != "drop" else 0)
        flops = 40 * 2 * (_grid_springs(n) if kind == "drop" else 3 * M)
        return {"bytes": substeps * step + 12 * obstacle + 60 * (V + obstacle // 2), "flops": substeps * flops}
    if kind == "batch":
        rng = np.random.Generator(np.random.PCG64(case["mix"]))  # the generator's draws, in its order
        V = S = 0
        for _ in range(case["instances"]):
            P = int(rng.integers(case["lo"], case["hi"] + 1))
            rng.uniform(0.2, 0.5), rng.uniform(-0.2, 0.2, 3), rng.uniform(0.0, 1e-4, P * P)
            V += P * P
            S += _grid_springs(P)
        substeps = 10 * case["frames"]
        return {"bytes": substeps * 68 * V + 60 * (V + 2562 * case["instances"]), "flops": substeps * 80 * S}
    if kind == "rollout":
        w = 2 if case["bits"] == 64 else 1
        V, S = case["side"] ** 2, _grid_springs(case["side"])
        # forward, its recomputation, and the reverse pass reading the state and updating the gradients
        return {"bytes": case["steps"] * w * (3 * (68 * V + 8 * S) + 16 * S), "flops": case["steps"] * 300 * S}
    if kind == "bvh":
        n = case["triangles"]
        return {"bytes": n * (36 + 12 + 72 + 8) + n * (72 + 12 + 64) + 64 * n + 12 * case["queries"], "flops": 0}
    if kind == "hash":
        n = case["triangles"]
        # triangles in, about two cell entries of 8 bytes each out and in again, queries in
        return {"bytes": n * 48 + 32 * n + 12 * case["queries"], "flops": 0}
    if kind == "facehash":
        M = 2 * (case["side"] - 1) ** 2 + 20 * 4 ** case["level"]
        return {"bytes": M * (12 + 6) + 50 * 32 * M, "flops": 0}
    return {"bytes": 16 * case["pairs"], "flops": 0}


# ------------------------------------------------------------------ the same in 64 bits
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.from_numpy(np.asarray(a)).to(_dev()).double()


class _Obstacle:
    """Static triangles of one mesh: corners, unit normals, boxes."""

    def __init__(self, x, facets):
        f = torch.from_numpy(facets.astype(np.int64)).to(x.device)
        self.t = x[f]
        self.lo, self.hi = self.t.amin(1), self.t.amax(1)
        self.root = x.amin(0), x.amax(0)
        self.facets = f


def _pairs(lo, hi, blo, bhi, limit=1 << 26):
    """(i, j) with box i of the first set meeting box j of the second, ascending."""
    out = []
    near = ((lo <= bhi.amax(0)) & (hi >= blo.amin(0))).all(1).nonzero()[:, 0] if len(blo) else lo.new_zeros(0).long()
    step = max(1, limit // max(1, len(blo)))
    for k in range(0, len(near), step):
        at = near[k:k + step]
        m = torch.ones(len(at), len(blo), dtype=torch.bool, device=lo.device)
        for a in range(3):
            m &= lo[at, a, None] <= bhi[None, :, a]
            m &= hi[at, a, None] >= blo[None, :, a]
        ij = m.nonzero()
        out.append(torch.stack([at[ij[:, 0]], ij[:, 1]], 1))
    return torch.cat(out) if out else torch.zeros(0, 2, dtype=torch.int64, device=lo.device)


def _dist2(p, t):
    """Squared distance of points to triangles (the closest of the interior's projection and the three edges)."""
    a, b, c = t[:, 0], t[:, 1], t[:, 2]
    def edge(u, w):
        d = w - u
        s = (((p - u) * d).sum(1) / (d * d).sum(1).clamp_min(1e-300)).clamp(0.0, 1.0)
        return ((p - u - s[:, None] * d) ** 2).sum(1)
    best = torch.minimum(torch.minimum(edge(a, b), edge(b, c)), edge(c, a))
    n = torch.linalg.cross(b - a, c - a)
    nn = (n * n).sum(1).clamp_min(1e-300)
    h = ((p - a) * n).sum(1)
    q = p - n * (h / nn)[:, None]
    inside = torch.ones_like(h, dtype=torch.bool)
    for u, w in ((a, b), (b, c), (c, a)):
        inside &= (torch.linalg.cross(w - u, q - u) * n).sum(1) >= 0
    return torch.where(inside, torch.minimum(best, h * h / nn), best)


def _contacts(x, xprev, t, band, thickness):
    """Of the candidate (point, triangle) rows those whose contact moves the point: mask, oriented normal."""
    e0, e1 = t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]
    n = torch.linalg.cross(e0, e1)
    nl2 = (n * n).sum(1)
    n = n / nl2.clamp_min(1e-300).sqrt()[:, None]
    dp, dc = ((xprev - t[:, 0]) * n).sum(1), ((x - t[:, 0]) * n).sum(1)
    flip = torch.where(dp != 0, dp, dc) < 0
    n = torch.where(flip[:, None], -n, n)
    dp, dc = torch.where(flip, -dp, dp), torch.where(flip, -dc, dc)
    cross = (dc < 0) & (dp > 0)
    s = torch.where(cross, dp / torch.where(cross, dp - dc, torch.ones_like(dp)), torch.ones_like(dp))
    pc = xprev + (x - xprev) * s[:, None] - t[:, 0]
    q = pc - n * (pc * n).sum(1, keepdim=True)
    d00, d01, d11 = (e0 * e0).sum(1), (e0 * e1).sum(1), (e1 * e1).sum(1)
    d20, d21 = (q * e0).sum(1), (q * e1).sum(1)
    den = d00 * d11 - d01 * d01
    b, c = (d11 * d20 - d01 * d21) / den, (d00 * d21 - d01 * d20) / den
    hit = (nl2 >= 1e-12) & (dc < band) & (den.abs() >= 1e-12) & (b >= 0) & (c >= 0) & (1 - b - c >= 0)
    return hit & (dc < thickness), n


def _grid_force(n, x, v, k, L, kd):
    """Spring forces of an n x n FastGridCloth with per-spring stiffness and rest length (canonical order)."""
    x, v, f = x.view(n, n, 3), v.view(n, n, 3), torch.zeros(n, n, 3, dtype=x.dtype, device=x.device)
    at = 0
    for (r0, c0), (r1, c1) in (((0, 0), (0, 1)), ((0, 0), (1, 0)), ((0, 0), (1, 1)), ((0, 1), (1, 0)), ((0, 0), (0, 2)),
                               ((0, 0), (2, 0))):
        h, w = n - max(r0, r1), n - max(c0, c1)
        ia, ib = (slice(r0, r0 + h), slice(c0, c0 + w)), (slice(r1, r1 + h), slice(c1, c1 + w))
        ks, Ls = k[at:at + h * w].view(h, w), L[at:at + h * w].view(h, w)
        at += h * w
        dx, dv = x[ib] - x[ia], v[ib] - v[ia]
        length = (dx * dx).sum(2).sqrt()
        d = dx / length[..., None]
        F = d * (ks * (length - Ls) + kd * (dv * d).sum(2))[..., None]
        pad = torch.nn.functional.pad
        f = f + pad(F, (0, 0, c0, n - c0 - w, r0, n - r0 - h)) - pad(F, (0, 0, c1, n - c1 - w, r1, n - r1 - h))
    return f.reshape(-1, 3)


def _mesh_springs(x, facets):
    """Stretch springs (edges) and bend springs (the two corners across an edge) of a triangle cloth: ends, lengths."""
    f = facets.astype(np.int64)
    e = np.concatenate([f[:, [0, 1, 2]], f[:, [1, 2, 0]], f[:, [2, 0, 1]]])
    lo, hi = np.minimum(e[:, 0], e[:, 1]), np.maximum(e[:, 0], e[:, 1])
    order = np.lexsort((hi, lo))
    lo, hi, opp = lo[order], hi[order], e[order, 2]
    new = np.concatenate([[True], (lo[1:] != lo[:-1]) | (hi[1:] != hi[:-1])])
    twin = np.nonzero(~new)[0]
    ends = [np.stack([lo[new], hi[new]], 1), np.stack([opp[twin - 1], opp[twin]], 1)]
    return [(torch.from_numpy(s).to(_dev()), torch.linalg.norm(_t(x)[s[:, 0]] - _t(x)[s[:, 1]], dim=1)) for s in ends]


def _mesh_force(springs, ks, x, v, kd):
    f = torch.zeros_like(x)
    for (s, rest), k in zip(springs, ks):
        a, b = s[:, 0], s[:, 1]
        dx, dv = x[b] - x[a], v[b] - v[a]
        length = (dx * dx).sum(1).sqrt()
        d = dx / length[:, None]
        F = d * (k * (length - rest) + kd * (dv * d).sum(1))[:, None]
        f = f.index_add(0, a, F).index_add(0, b, -F)
    return f


def _substep(prm, cloth, force, obst, x, xprev, v, facets=None):
    """One substep of a cloth over a static obstacle: candidates, contacts, forces, response, integration."""
    h, mass, gravity = prm["subh"], prm["mass"], torch.tensor(prm["gravity"], dtype=x.dtype, device=x.device)
    with torch.no_grad():
        rows, margin = [], prm["margin"]
        if facets is not None:
            t = x[facets]
            if prm["self_mode"] == 1:
                lo, hi = torch.minimum(x, xprev), torch.maximum(x, xprev)
                ij = _pairs(lo, hi, t.amin(1) - margin, t.amax(1) + margin)
            else:
                u = t + v[facets] * h
                ij = _pairs(x - margin, x + margin, torch.minimum(t, u).amin(1), torch.maximum(t, u).amax(1))
            ij = ij[(facets[ij[:, 1]] != ij[:, :1]).all(1)]
            if prm["self_mode"] == 1:
                tt = t[ij[:, 1]]
                ij = ij[(_dist2(x[ij[:, 0]], tt) <= margin ** 2) | (_dist2(xprev[ij[:, 0]], tt) <= margin ** 2)]
            rows.append((ij, t[ij[:, 1]]))
        u = x + v * h
        root = torch.minimum(x, u).amin(0), torch.maximum(x, u).amax(0)
        if bool(((root[0] <= obst.root[1]) & (root[1] >= obst.root[0])).all()):
            ij = _pairs(x - margin, x + margin, obst.lo, obst.hi)
            rows.append((ij, obst.t[ij[:, 1]]))
        hits = []
        for ij, t in rows:
            hit, n = _contacts(x[ij[:, 0]], xprev[ij[:, 0]], t, prm["band"], prm["thickness"])
            hits.append((ij[hit, 0], n[hit], t[hit, 0]))
        point = torch.cat([p for p, _, _ in hits]) if hits else torch.zeros(0, dtype=torch.int64, device=x.device)
    v = v + (gravity * mass + v * prm["kair"] + force(x, v)) * (h / mass)
    pos = x
    if len(point):
        # a point's contacts act one after another, self rows first, by ascending triangle
        order = torch.sort(point, stable=True).indices
        point = point[order]
        n, t0 = torch.cat([q for _, q, _ in hits])[order], torch.cat([q for _, _, q in hits])[order]
        first = torch.searchsorted(point, point)
        rank = torch.arange(len(point), device=x.device) - first
        for r in range(int(rank.max()) + 1):
            at = rank == r
            p, nn = point[at], n[at]
            vn = (v[p] * nn).sum(1)
            v = v.index_add(0, p, nn * (-vn.clamp_max(0.0))[:, None])
            pos = pos.index_add(0, p, nn * (prm["thickness"] - ((x[p] - t0[at]) * nn).sum(1))[:, None])
    return pos + v * h, x, v


def _params(spec, m):
    p, f = spec.params, lambda a: float(np.float32(a))
    return {"subh": f(p.subh), "mass": f(m.mass[0]), "gravity": [f(g) for g in p.gravity], "margin": f(p.margin),
            "band": f(np.float32(p.radius) + np.float32(p.margin)), "thickness": f(m.thickness), "kair": f(p.kair),
            "kd": f(p.kd), "self_mode": p.self_mode}


def _run_cloth(spec, m, obst, steps, x, xprev, v, k=None, L=None, facets=None):
    prm = _params(spec, m)
    if m.grid_n:
        if k is None:
            k, L = (_t(a) for a in G.grid_spring_params(m.grid_n, m.grid_rest, (m.kstretch, m.kshear, m.kbend)))
        def force(x, v):
            return _grid_force(m.grid_n, x, v, k, L, prm["kd"])
    else:
        springs = _mesh_springs(m.x, m.facets)
        def force(x, v):
            return _mesh_force(springs, (float(m.kstretch), float(m.kbend)), x, v, prm["kd"])
    for _ in range(steps):
        x, xprev, v = _substep(prm, m, force, obst, x, xprev, v, facets)
    return x, v


def exact(case, seed):
    """The same episodes and rollouts in binary64, every point against every triangle.  The drape's start state is a
    result of stepping, and the other kinds return whole numbers."""
    kind = case["kind"]
    if kind == "rollout":
        spec, k, L, v0, target = _rollout(case, seed)
        m, o = spec.meshes
        k, L, v0 = (_t(a).requires_grad_() for a in (k, L, v0))
        x0 = _t(m.x)
        x, _ = _run_cloth(spec, m, _Obstacle(_t(o.x), o.facets), case["steps"], x0, x0, v0, k, L)
        loss = ((x - _t(target)) ** 2).sum(1).mean()
        gk, gL, gv = torch.autograd.grad(loss, (k, L, v0))
        return {"x": x.detach(), "gk": gk, "gL": gL, "gv": gv}
    if kind not in ("drop", "fold", "batch") or case["frames"] * case.get("instances", 1) > 480:
        return None
    spec, start = _scene(case, seed)
    xs, xp, vs = (_t(start[w]) for w in ("x", "xprev", "v"))
    at, steps = 0, case["frames"] * spec.params.substeps
    for m, o in zip(spec.meshes[0::2], spec.meshes[1::2]):
        c, ob = slice(at, at + m.nV), slice(at + m.nV, at + m.nV + o.nV)
        facets = torch.from_numpy(m.facets.astype(np.int64)).to(_dev()) if kind == "fold" else None
        xs[c], vs[c] = _run_cloth(spec, m, _Obstacle(xs[ob], o.facets), steps, xs[c].clone(), xp[c].clone(),
                                  vs[c].clone(), facets=facets)
        at += m.nV + o.nV
    return {"x": xs, "v": vs, "rows": None, "contacts": None, "flags": None}
