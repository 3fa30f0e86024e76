"""A workspace, plan or context made for many items serves any smaller number
of them, on both sides of every size where the sorts change their tiles."""
import ctypes

import numpy as np
import pytest

from gtc import workloads as W

# The sorts' short tiles end at these key counts (1,024 and 2,048 keys a tile).
SORT_LIMITS = (160 * 1024, 200 * 2048)


def sizes_around(limits):
    n = set(range(1, 1_400_000, 3_001))
    for x in limits:
        n.update(range(max(x - 70_000, 1), x + 70_000, 257))
        n.update((x - 1, x, x + 1))
    return sorted(n)


@pytest.mark.parametrize("op,key_bits", [(op, kb) for op in ("SORT_PAIRS", "GLOBAL_HISTOGRAM", "UNIQUE", "PARTIAL_SUM",
                                                             "BUILD_OCTREE", "LEARNED_SORT")
                                         for kb in (32, 64) if (op, kb) != ("LEARNED_SORT", 32)])
def test_workspace_never_shrinks(gtc_mod, op, key_bits):
    code = getattr(gtc_mod, "OP_" + op)
    b, last = ctypes.c_size_t(), (0, 0)
    for n in sizes_around(SORT_LIMITS):
        assert gtc_mod.lib().gtc_workspace_size(None, code, n, key_bits, ctypes.byref(b)) == 0
        assert b.value >= last[1], (n, last)
        last = (n, b.value)


@pytest.mark.parametrize("clouds", [1, 16, 64, 1000])
def test_batched_workspace_never_shrinks(gtc_mod, clouds):
    b, last = ctypes.c_size_t(), (0, 0)
    for n in sizes_around((600_000,)):
        assert gtc_mod.lib().gtc_batched_workspace_size(n, clouds, ctypes.byref(b)) == 0
        assert b.value >= last[1], (n, last)
        last = (n, b.value)


# (capacity, items): the items' own workspace has more tiles than the capacity's.
REUSE = [(170_000, 160_000), (180_000, 163_840), (190_000, 163_841), (420_000, 400_000), (440_000, 409_600),
         (440_000, 409_601)]


@pytest.mark.gpu
@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("cap,n", REUSE)
def test_plan_with_fewer_points(gtc_mod, oracle, key_bits, cap, n):
    import torch

    from test_gpu_pipeline import _cmp

    c = gtc_mod.Context(0)
    plan = gtc_mod.OctreePlan(c, cap, key_bits)
    for m, seed in ((cap, 1), (n, 2)):
        pts = W.gaussian_mixture_points(m, 8, 10.0, noise=0.2, seed=seed)
        plan.launch(torch.from_numpy(pts).cuda())
        _cmp(plan.result(), oracle.build_octree(pts, key_bits, threads=8)[0], key_bits, (cap, m))
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("queued", [False, True])
def test_host_frames_of_varying_size(gtc_mod, oracle, queued):
    """Frames through one context, each into page-locked memory of its own."""
    import torch

    c = gtc_mod.Context(0)
    jobs = []
    for n in [m for pair in REUSE for m in (pair[0], pair[0], pair[1], pair[1])]:  # both queue slots
        pts = torch.from_numpy(W.gaussian_mixture_points(n, 8, 10.0, noise=0.2, seed=n)).pin_memory()
        jobs.append((pts, torch.zeros((2 * n, 16), dtype=torch.int32).pin_memory(),
                     torch.zeros(4, dtype=torch.int32).pin_memory()))
    for pts, nodes, counts in jobs:
        f = c.L.gtc_build_octree_host_async if queued else c.L.gtc_build_octree_host
        c.check(f(c.h, pts.data_ptr(), pts.shape[0], 0.0, 1024.0, 64, nodes.data_ptr(), nodes.shape[0],
                  counts.data_ptr()))
    if queued:
        c.check(c.L.gtc_build_octree_host_wait(c.h))
    c.close()
    for pts, nodes, counts in jobs:
        exp, _ = oracle.build_octree(pts.numpy(), 64, threads=8)
        o = exp["n_oct_nodes"]
        assert counts[:3].tolist() == [exp["n_unique"], exp["n_brt_nodes"], o]
        assert np.array_equal(nodes[:o].numpy(), exp["nodes"].view(np.int32).reshape(o, 16))


@pytest.mark.gpu
@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("cap,n", [(200_000, 163_840), (325_000, 163_840), (500_000, 163_840), (500_000, 409_600)])
def test_sort_with_a_larger_workspace(gtc_mod, key_bits, cap, n):
    """The caller's workspace, and the context's own under capture: warmed up
    by a larger sort, a smaller one must not allocate."""
    import torch

    td = np.int32 if key_bits == 32 else np.int64
    c = gtc_mod.Context(0)
    src = torch.from_numpy(W.config3_keys(n, key_bits, seed=cap).view(td)).cuda()
    want = np.sort(src.cpu().numpy().view(np.uint32 if key_bits == 32 else np.uint64)).view(td)
    k, alt = src.clone(), torch.empty_like(src)
    c.sort_pairs(k, None, ws=c.workspace(gtc_mod.OP_SORT_PAIRS, cap, key_bits), keys_alt=alt)
    assert np.array_equal(k.cpu().numpy(), want)

    big = torch.from_numpy(W.config3_keys(cap, key_bits, seed=n).view(td)).cuda()
    c.sort_pairs(big, None)
    torch.cuda.synchronize()
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(s):
        g.capture_begin()
        c.sort_pairs(k, None, keys_alt=alt)
        g.capture_end()
    k.copy_(src)
    g.replay()
    assert np.array_equal(k.cpu().numpy(), want)
    assert c.device_status() == 0
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cap,n", [(184_000, 163_840), (436_000, 409_600)])
def test_learned_sort_with_a_larger_workspace(gtc_mod, cap, n):
    import torch

    c = gtc_mod.Context(0)
    keys = torch.from_numpy(W.config3_keys(n, 64, seed=n).view(np.int64)).cuda()
    prior = keys.clone()
    c.sort_pairs(prior)
    model = gtc_mod.LearnedModel(c, gtc_mod.learned_buckets_for(n))
    model.train(prior, stride=10)
    out = model.sort(keys, ws=c.workspace(gtc_mod.OP_LEARNED_SORT, cap, 64))
    assert torch.equal(out[0], prior)
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cap,clouds_cap,n,clouds", [(600_001, 16, 600_000, 16), (640_000, 16, 600_000, 16),
                                                     (640_000, 64, 599_999, 63), (640_000, 64, 600_001, 64)])
def test_batch_plan_with_fewer_points(gtc_mod, oracle, cap, clouds_cap, n, clouds):
    import torch

    from test_gpu_pipeline import _cmp

    c = gtc_mod.Context(0)
    plan = gtc_mod.BatchPlan(c, cap, clouds_cap)
    for m, s in ((cap, clouds_cap), (n, clouds)):
        off = np.linspace(0, m, s + 1).astype(np.int64)
        pts = W.gaussian_mixture_points(m, 8, 10.0, noise=0.2, seed=m + s)
        plan.launch(torch.from_numpy(pts).cuda(), torch.from_numpy(off.astype(np.int32)).cuda())
        for k, r in enumerate(plan.clouds()):
            exp, _ = oracle.build_octree(np.ascontiguousarray(pts[off[k]:off[k + 1]]), 32, threads=8)
            _cmp(r, exp, 32, (m, k))
    c.close()
