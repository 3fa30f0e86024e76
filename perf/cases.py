"""The work that users of the library have it do, as cases that can be timed.

A case is a call, or the short sequence of calls that a program makes, on one
point cloud, key set or batch: its sizes are those of the benchmark, of the
tests and of the named workloads (gtc/workloads.py), and odd ones between
them.  Every output is a whole number or, in the octree nodes, a bit pattern
(an octree node is 16 words: child indices, masks, and the corner and cell
size as float bits), and every result is defined exactly: the stable sort and
the tree of the sorted codes.  So no output is held to a tolerance, and no
64-bit value is given beside it.

Inputs are drawn on the GPU from the seed; the distributions are those of
gtc/workloads.py: uniform points, Gaussian mixtures with uniform noise, keys
that are ANDs of uniform words.  A tree's arrays are as long as its cloud has
distinct codes and octree nodes, so a case's clouds are one drawn cloud,
flipped by the seed in random bits of its cell coordinates (_flip): other
codes, order and tree, with the same number of codes and nodes.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("glsl-tree-construction_gb300"))

import gtc  # noqa: E402
from gtc import workloads as W  # noqa: E402

DEV = "cuda:0"
RANGE = 1024.0
TOP = float(np.nextafter(np.float32(RANGE), np.float32(0.0)))

_ctx = None


def ctx():
    """The program's one context, made at its first use."""
    global _ctx
    if _ctx is None:
        _ctx = gtc.Context(0)
    return _ctx


# ------------------------------------------------------------------ cases --

def listed():
    return [
        # One small cloud after another, as from a depth sensor's sub-map: the
        # build is a handful of short dependent launches.
        {"name": "small_u32", "kind": "build", "n": 4096, "bits": 32, "cloud": "uniform", "graph": False},
        # One LiDAR sweep of ragged size with full-depth codes.
        {"name": "sweep_u64", "kind": "build", "n": 120_007, "bits": 64, "cloud": "mixture", "graph": False},
        # The plain pipeline's uniform million-point cloud, 32-bit codes.
        {"name": "uniform_1m_u32", "kind": "build", "n": 1 << 20, "bits": 32, "cloud": "uniform", "graph": False},
        # The headline build: 10M clustered points, 64-bit codes, replayed as a
        # captured graph, as the benchmark does it.
        {"name": "clustered_10m_u64", "kind": "build", "n": 10_000_000, "bits": 64, "cloud": "mixture",
         "graph": True},
        # Stage by stage, as the reference's main program calls its operators:
        # the host reads the unique and node counts between stages.
        {"name": "stages_1m_u64", "kind": "stages", "n": 1_000_003, "bits": 64, "cloud": "uniform"},
        # Points and nodes in page-locked host memory, one build at a time.
        {"name": "host_1m_u64", "kind": "host", "n": 1 << 20, "bits": 64, "cloud": "mixture"},
        # Many clouds of 1K to 1M points in one captured batch.
        {"name": "batch_512", "kind": "batch", "clouds": 512, "lo": 1000, "hi": 1_000_000, "graph": True},
        # A batch of small clouds (objects or tiles of a scene), launched anew.
        {"name": "batch_small", "kind": "batch", "clouds": 64, "lo": 300, "hi": 20_000, "graph": False},
        # Sort of key-value pairs: the sweep's small end, a ragged middle size
        # of 64-bit keys with low-entropy digits, and its usual large size.
        {"name": "sort_64k_u32", "kind": "sort", "n": 1 << 16, "bits": 32, "ands": 0},
        {"name": "sort_3m_u64", "kind": "sort", "n": 3_000_017, "bits": 64, "ands": 2},
        {"name": "sort_16m_u32", "kind": "sort", "n": 1 << 24, "bits": 32, "ands": 0},
        # The learned-bucket sort of 64M Morton keys with a model trained on an
        # earlier sample of the same mixture.
        {"name": "learned_64m", "kind": "learned", "n": 1 << 26},
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["build", "build", "build", "sort", "sort", "stages", "host", "batch", "batch", "learned"])
    if kind == "build":
        return {"kind": kind, "n": _log(rng, 256, 10_000_000), "bits": rng.choice([32, 64]),
                "cloud": rng.choice(["uniform", "mixture"]), "graph": rng.random() < 0.5}
    if kind in ("stages", "host"):
        return {"kind": kind, "n": _log(rng, 1000, 4_000_000), "bits": rng.choice([32, 64]),
                "cloud": rng.choice(["uniform", "mixture"])}
    if kind == "sort":
        return {"kind": kind, "n": _log(rng, 1 << 10, 1 << 25), "bits": rng.choice([32, 64]),
                "ands": rng.choice([0, 0, 1, 2, 3, 4])}
    if kind == "batch":
        lo = _log(rng, 200, 20_000)
        case = {"kind": kind, "clouds": _log(rng, 2, 512), "lo": lo, "hi": lo * rng.randint(1, 40),
                "graph": rng.random() < 0.5}
        while _batch_offsets(case)[-1] > 80_000_000:
            case["clouds"] = case["clouds"] * 2 // 3
        return case
    return {"kind": kind, "n": _log(rng, 1 << 22, 1 << 26)}


# ----------------------------------------------------------------- inputs --

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _pack(xyz):
    pts = torch.ones((xyz.shape[0], 4), dtype=torch.float32, device=DEV)
    pts[:, :3] = xyz
    return pts


def _mixture(g, comp, centres, sigma, noise):
    """Gaussian mixture points around centres[comp] with `noise` of uniform
    ones, clamped below the top of the domain."""
    n = comp.shape[0]
    xyz = centres[comp] + torch.randn((n, 3), generator=g, device=DEV) * sigma[comp].unsqueeze(1)
    if noise > 0.0:
        u = torch.rand((n, 3), generator=g, device=DEV) * RANGE
        xyz = torch.where(torch.rand((n, 1), generator=g, device=DEV) < noise, u, xyz)
    return xyz.clamp_(0.0, TOP)


def _flip(xyz, seed, clouds=1, cloud=None):
    """The points with the 21-bit cell coordinates of each cloud XORed by a
    random mask: cells that agree in their leading bits still do, so the octree
    is the same up to the order of its octants.  Points keep 3 bits inside
    their cell, so that every coordinate is an exact float32."""
    mask = torch.randint(0, 1 << 21, (clouds, 3), generator=_gen(seed), device=DEV, dtype=torch.int32)
    q = (xyz * (8.0 * 2048.0)).to(torch.int32)
    q ^= (mask if cloud is None else mask[cloud]) << 3
    return q.to(torch.float32) * (1.0 / (8.0 * 2048.0))


def _cloud(n, cloud, seed):
    """Uniform points, or 32 clusters of sigma 0.5% of the domain with 2% noise."""
    g = _gen(n)
    if cloud == "uniform":
        xyz = torch.rand((n, 3), generator=g, device=DEV) * RANGE
    else:
        centres = torch.rand((32, 3), generator=g, device=DEV) * RANGE
        comp = torch.randint(0, 32, (n,), generator=g, device=DEV)
        xyz = _mixture(g, comp, centres, torch.full((32,), 0.005 * RANGE, device=DEV), 0.02)
    return _pack(_flip(xyz, seed))


def _batch_offsets(case):
    """Log-uniform cloud sizes in a fixed shuffled order (the seed moves the
    points, not the sizes)."""
    s, lo, hi = case["clouds"], case["lo"], case["hi"]
    sizes = (lo * (hi / lo) ** ((np.arange(s) + 0.5) / s)).astype(np.int64)
    sizes = sizes[np.random.Generator(np.random.PCG64(11)).permutation(s)]
    return np.concatenate([[0], np.cumsum(sizes)])


def _batch_points(off, seed):
    """Even clouds uniform, odd clouds 8 clusters of sigma 1% of the domain."""
    s, n = off.shape[0] - 1, int(off[-1])
    g = _gen(n)
    sizes = torch.from_numpy(np.diff(off)).to(DEV)
    cloud = torch.repeat_interleave(torch.arange(s, device=DEV), sizes, output_size=n)
    centres = torch.rand((s * 8, 3), generator=g, device=DEV) * RANGE
    comp = cloud * 8 + torch.randint(0, 8, (n,), generator=g, device=DEV)
    xyz = _mixture(g, comp, centres, torch.full((s * 8,), 0.01 * RANGE, device=DEV), 0.0)
    u = torch.rand((n, 3), generator=g, device=DEV) * RANGE
    return _pack(_flip(torch.where((cloud % 2 == 0).unsqueeze(1), u, xyz), seed, s, cloud))


def _words(n, bits, ands, g):
    """Uniform words, or the AND of `ands` of them (bit density 2^-ands)."""
    k = None
    for _ in range(max(ands, 1)):
        r = torch.randint(-(1 << (bits - 1)), (1 << (bits - 1)) - 1, (n,), generator=g, device=DEV,
                          dtype=torch.int64)
        k = r if k is None else k & r
    return k.to(torch.int32) if bits == 32 else k


def _learned_points(n, seed):
    """The learned sort's fixed 64-component mixture; the seed draws the sample."""
    g = np.random.Generator(np.random.PCG64(10_000))
    centres = torch.from_numpy((g.random((64, 3)) * W.DOMAIN_RANGE).astype(np.float32)).to(DEV)
    sigma = torch.from_numpy((g.uniform(0.003, 0.03, 64) * W.DOMAIN_RANGE).astype(np.float32)).to(DEV)
    weight = torch.from_numpy(g.exponential(1.0, 64)).to(DEV)
    edge = torch.cumsum(weight / weight.sum(), 0)
    t = _gen(seed)
    comp = torch.searchsorted(edge, torch.rand(n, generator=t, device=DEV, dtype=torch.float64)).clamp_(max=63)
    return _pack(_mixture(t, comp, centres, sigma, 0.05))


class Build:
    """A cloud and the plan that builds it; `launch` is one build."""

    def __init__(self, case, seed):
        self.pts = _cloud(case["n"], case["cloud"], seed)
        self.plan = gtc.OctreePlan(ctx(), case["n"], case["bits"])
        if case["graph"]:
            self.plan.capture(self.pts)
        else:
            self.plan.launch(self.pts)
        self.graph = case["graph"]
        r = self.plan.result()  # the live lengths, so that a pass need not read them back
        self.out = {f: getattr(r, f) for f in gtc.STAGE_BUFFERS}
        self.out["counts"] = self.plan.counts

    def run(self):
        if self.graph:
            self.plan.replay()
        else:
            self.plan.launch(self.pts)
        return self.out


class Stages:
    """The stage operators in the order of the reference's main program."""

    def __init__(self, case, seed):
        self.bits, self.n = case["bits"], case["n"]
        self.pts = _cloud(self.n, case["cloud"], seed)
        self.ws = ctx().workspace(gtc.OP_SORT_PAIRS, self.n, self.bits)
        self.scan_ws = ctx().workspace(gtc.OP_UNIQUE, self.n, self.bits)

    def run(self):
        c, bits = ctx(), self.bits
        keys, idx = c.morton(self.pts, bits)
        c.sort_pairs(keys, idx, 0, 30 if bits == 32 else 63, ws=self.ws)
        u = int(c.unique(keys, idx, ws=self.scan_ws).item())
        codes = keys[:u]
        tree = c.radix_tree(codes, u - 1)
        edge = c.edge_count(tree["prefix_n"], tree["parent"], bits)
        ps, o = c.node_offsets(edge, u - 1, ws=self.scan_ws)
        nodes = c.make_octree(codes, tree, edge, ps, int(o.item()))
        pts = c.gather_points(self.pts, idx, u)
        return {"codes": codes, "idx": idx[:u], **tree, "edge_count": edge, "node_offsets": ps, "nodes": nodes,
                "points": pts.view(torch.int32)}


class Host:
    """A cloud in page-locked host memory, its nodes read back to the host."""

    def __init__(self, case, seed):
        self.n, self.bits = case["n"], case["bits"]
        self.pts = _cloud(self.n, case["cloud"], seed).cpu().pin_memory()
        self.cap = self.n + 1024
        self.nodes = torch.zeros((self.cap, 16), dtype=torch.int32).pin_memory()
        self.counts = torch.zeros(4, dtype=torch.int32).pin_memory()

    def run(self):
        c = ctx()
        c.check(c.L.gtc_build_octree_host(c.h, self.pts.data_ptr(), self.n, 0.0, RANGE, self.bits,
                                          self.nodes.data_ptr(), self.cap, self.counts.data_ptr()))
        return {"nodes": self.nodes[: int(self.counts[2])], "counts": self.counts[:3]}


class Batch:
    """Many clouds and the plan that builds them in one sequence of launches."""

    def __init__(self, case, seed):
        off = _batch_offsets(case)
        self.pts = _batch_points(off, seed)
        self.off = torch.from_numpy(off.astype(np.uint32).view(np.int32)).to(DEV)
        self.plan = gtc.BatchPlan(ctx(), int(off[-1]), case["clouds"])
        if case["graph"]:
            self.plan.capture(self.pts, self.off)
        else:
            self.plan.launch(self.pts, self.off)
        self.graph = case["graph"]
        ctx().device_status()
        # Every cloud's outputs follow each other, so the batch's live lengths
        # are one slice per array.  The tree arrays hold one entry per cloud
        # that no build writes (a cloud of u codes has u - 1 radix nodes): 0 here.
        p = self.plan
        tree = {"prefix_n": p.prefix_n, "has_leaf_left": p.hll, "has_leaf_right": p.hlr, "left_child": p.left,
                "parent": p.parent, "edge_count": p.edge}
        for t in tree.values():
            t.zero_()
        ko, no, _ = p.host_offsets()
        u, o = int(ko[-1]), int(no[-1])
        self.out = {"keys": p.keys[:u], "idx": p.idx[:u], "node_offsets": p.ps[:u], "nodes": p.nodes[:o],
                    "key_offset": p.key_offset, "node_offset": p.node_offset, "cloud_counts": p.cloud_counts}
        self.out.update({f: t[:u] for f, t in tree.items()})

    def run(self):
        if self.graph:
            self.plan.replay()
        else:
            self.plan.launch(self.pts, self.off)
        return self.out


class Sort:
    """Key-value pairs that arrive in the caller's buffers and are sorted in
    place in a kept pair of work buffers."""

    def __init__(self, case, seed):
        n, bits = case["n"], case["bits"]
        self.keys_in = _words(n, bits, case["ands"], _gen(seed))
        self.vals_in = torch.arange(n, dtype=torch.int32, device=DEV)
        self.keys, self.vals = torch.empty_like(self.keys_in), torch.empty_like(self.vals_in)
        self.alt = torch.empty_like(self.keys_in), torch.empty_like(self.vals_in)
        self.ws = ctx().workspace(gtc.OP_SORT_PAIRS, n, bits)

    def run(self):
        self.keys.copy_(self.keys_in)
        self.vals.copy_(self.vals_in)
        return ctx().sort_pairs(self.keys, self.vals, ws=self.ws, keys_alt=self.alt[0], vals_alt=self.alt[1])


class Learned:
    """64-bit Morton keys of one sample, sorted with a model trained on an
    earlier, sorted sample of the same mixture."""

    def __init__(self, case, seed):
        c, n = ctx(), case["n"]
        prior = c.morton(_learned_points(n, 77), 64, with_idx=False)[0]
        c.sort_pairs(prior)
        self.model = gtc.LearnedModel(c, gtc.learned_buckets_for(n))
        self.model.train(prior)
        self.keys = c.morton(_learned_points(n, seed), 64, with_idx=False)[0]
        self.keys_out = torch.empty_like(self.keys)
        self.vals_out = torch.empty(n, dtype=torch.int32, device=DEV)
        self.ws = c.workspace(gtc.OP_LEARNED_SORT, n, 64)

    def run(self):
        return self.model.sort(self.keys, ws=self.ws, keys_out=self.keys_out, vals_out=self.vals_out)


KINDS = {"build": Build, "stages": Stages, "host": Host, "batch": Batch, "sort": Sort, "learned": Learned}


def prepare(case, seed):
    return KINDS[case["kind"]](case, seed)


def run(state):
    return state.run()


def work(case):
    """Bytes of one pass: the inputs read once and the outputs written once,
    with nearly every code distinct and half as many octree nodes as points.
    The arithmetic is integer; no floating-point work is counted."""
    kind = case["kind"]
    n = int(_batch_offsets(case)[-1]) if kind == "batch" else case["n"]
    k = case.get("bits", 32) // 8
    nodes = 32 * n
    if kind == "sort":
        b = 2 * (k + 4) * n
    elif kind == "learned":
        b = (8 + 12) * n
    elif kind == "host":
        b = 16 * n + nodes
    else:  # points; codes, index, offsets; the tree's 3 bytes and 2 words and the edge counts; nodes
        b = 16 * n + (k + 8) * n + 15 * n + nodes
        if kind == "stages":
            b += 32 * n  # the points in sorted order
    return {"bytes": b, "flops": 0}
