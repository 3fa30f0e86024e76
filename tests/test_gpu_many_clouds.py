"""Batches of very many clouds, tiny and empty ones: every cloud's offsets and
outputs, and what a run of empty clouds costs."""
import numpy as np
import pytest

from gtc import workloads as W

pytestmark = pytest.mark.gpu


def build(ctx, gtc_mod, sizes, seed):
    import torch

    off = np.concatenate(([0], np.cumsum(sizes))).astype(np.int64)
    pts = W.uniform_points(int(off[-1]), seed=seed)
    plan = gtc_mod.BatchPlan(ctx, pts.shape[0], len(sizes))
    d = torch.from_numpy(pts).cuda(), torch.from_numpy(off.astype(np.int32)).cuda()
    plan.launch(*d)
    ctx.device_status()
    return plan, d, pts, off


def layout(name):
    g = np.random.Generator(np.random.PCG64(3))
    sizes = np.zeros(20_000, np.int64)
    if name == "tiny":
        return g.integers(1, 5, sizes.size)
    if name == "tiny_and_empty":
        return g.integers(0, 5, sizes.size)
    if name == "ones":
        return np.ones(sizes.size, np.int64)
    if name == "first":  # empty clouds first
        sizes[-40:] = 3001
    elif name == "last":
        sizes[:40] = 3001
    elif name == "middle":
        sizes[:20] = sizes[-20:] = 3001
    elif name == "runs":  # runs of empty clouds that start and end inside a row of 32 codes
        at = np.sort(g.choice(sizes.size, 400, replace=False))
        sizes[at] = g.integers(1, 70, 400)
    elif name == "segments":  # long enough for the segment form, and for groups of tiles
        sizes[::50] = 15_003
        sizes[10_000:12_000] = 0
    return sizes


@pytest.mark.parametrize("name", ["tiny", "tiny_and_empty", "ones", "first", "last", "middle", "runs", "segments"])
def test_many_clouds(ctx, gtc_mod, oracle, name):
    """Every cloud's unique codes, first indices and place against numpy; the
    tree and the octree of some clouds against the oracle."""
    from test_gpu_pipeline import _cmp

    sizes = layout(name)
    plan, _, pts, off = build(ctx, gtc_mod, sizes, seed=len(name))
    cloud = np.repeat(np.arange(sizes.size), sizes)
    codes = oracle.morton(pts, 32).astype(np.uint64) | (cloud.astype(np.uint64) << np.uint64(32))
    want, first = np.unique(codes, return_index=True)
    ko, no, cc = plan.host_offsets()
    assert np.array_equal(ko, np.searchsorted(want >> np.uint64(32), np.arange(sizes.size + 1)))
    assert np.array_equal(cc[:, 0], np.diff(ko)) and np.array_equal(cc[:, 1], np.maximum(cc[:, 0] - 1, 0))
    assert np.array_equal(np.diff(no), cc[:, 2])
    assert np.array_equal(plan.keys[:want.size].cpu().numpy().view(np.uint32), want.astype(np.uint32))
    assert np.array_equal(plan.idx[:want.size].cpu().numpy(), first - off[cloud[first]])
    res = plan.clouds()
    full = np.flatnonzero(sizes)
    for c in np.unique(np.concatenate((full[:3], full[-3:], full[:: max(full.size // 20, 1)]))):
        exp, _ = oracle.build_octree(np.ascontiguousarray(pts[off[c]:off[c + 1]]), 32)
        _cmp(res[c], exp, 32, (name, int(c)))


def test_a_run_of_empty_clouds_costs_little(ctx, gtc_mod):
    """100,000 slots, 100 of them with 3,000 points: in one place or spread,
    the batch is the same work.  A step per empty cloud, one dependent load
    each, would be 17 times that."""
    import torch

    def ms(at):
        sizes = np.zeros(100_000, np.int64)
        sizes[at] = 3_000
        plan, d, _, _ = build(ctx, gtc_mod, sizes, seed=1)
        a, b = torch.cuda.Event(True), torch.cuda.Event(True)
        t = []
        for _ in range(8):
            a.record()
            plan.launch(*d)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        return min(t)

    spread = ms(np.arange(0, 100_000, 1_000))
    for at in (np.arange(100), np.arange(99_900, 100_000), np.r_[0:50, 99_950:100_000]):
        assert ms(at) < 5 * spread
