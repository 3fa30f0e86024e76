"""Sizes at which a kernel's launch shape changes or a tile ends: one
parametrised test per dispatch rule, against the oracle or the other method
that the repository has for the same stage (bit-exact)."""
import numpy as np
import pytest

from gtc import workloads as W

pytestmark = pytest.mark.gpu


def unique_codes(oracle, n, key_bits, seed):
    """About n sorted distinct codes of a cloud with dense clusters (long and
    short ranges, three prefix lengths per depth band)."""
    pts = W.gaussian_mixture_points(n + n // 2 + 64, 5, 40.0, noise=0.3, seed=seed)
    codes = np.unique(oracle.morton(pts, key_bits))
    assert codes.size >= n
    return np.ascontiguousarray(codes[:n])


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("u", [2, 511, 512, 513, 514, 1025, 1026, 4097, 9000, 155_649, 155_650, 233_473, 233_474,
                               466_945, 466_946, 700_001, 700_002, 778_241, 778_242, 933_889, 933_890, 1_089_537,
                               1_089_538, 1_245_185, 1_245_186, 1_400_833, 1_400_834, 1_634_305, 1_634_306,
                               1_867_777, 1_867_778])
def test_tree_window_shapes(ctx, gtc_mod, oracle, key_bits, u):
    """u codes (u - 1 splits) at the tile edges and on both sides of the shape
    rule: the window method against the per-node search."""
    import torch

    codes = unique_codes(oracle, u, key_bits, seed=u)
    d = torch.from_numpy(codes.view(np.int32 if key_bits == 32 else np.int64)).cuda()
    L = gtc_mod.lib()
    got = ctx.radix_tree(d, u - 1, with_edge=True)
    try:
        assert L.gtc_tree_set_method(0) == 0
        want = ctx.radix_tree(d, u - 1, with_edge=True)
    finally:
        L.gtc_tree_set_method(1)
    assert ctx.device_status() == 0
    for f in want:
        assert torch.equal(got[f], want[f]), f


def small_clouds(n):
    """Clouds of n points that take the one-block build's paths: spread and
    clustered codes, one or few distinct codes, and runs of codes equal in
    their top 32 bits around the length one thread sorts (16) and far over."""
    g = np.random.Generator(np.random.PCG64(n))
    uniform = W.uniform_points(n, seed=n)
    yield "uniform", uniform
    yield "clusters", W.gaussian_mixture_points(n, 3, 2.0, noise=0.1, seed=n)
    yield "tight", W.gaussian_mixture_points(n, 1, 0.002, noise=0.002, seed=n)  # long runs
    yield "equal", np.tile(uniform[:1], (n, 1))
    yield "few", uniform[g.integers(0, min(n, 7), n)]
    side = 1024.0 / (1 << 11)  # a cell of the top 33 bits holds at most two runs
    for per in (15, 17):
        corner = np.floor(g.random((n // per + 1, 3)) * (1 << 11)) * side
        cube = uniform.copy()
        cube[:, :3] = np.repeat(corner, per, axis=0)[:n] + g.random((n, 3)) * side
        cube[:, :3] = np.minimum(cube[:, :3], 1023.99)
        yield f"runs_{per}", cube[g.permutation(n)]


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097])
def test_one_block_build(ctx, gtc_mod, oracle, key_bits, n):
    """One block up to 4,096 points, the stage kernels above: every output
    against the oracle, also under capture and at a node capacity one short."""
    import torch

    from test_gpu_pipeline import _cmp

    for name, pts in small_clouds(n):
        d = torch.from_numpy(pts).cuda()
        exp, _ = oracle.build_octree(pts, key_bits)
        plan = gtc_mod.OctreePlan(ctx, n, key_bits, nodes_capacity=exp["n_oct_nodes"])
        plan.launch(d)
        _cmp(plan.result(), exp, key_bits, (name, n))
        plan.nodes.zero_()
        plan.capture(d)
        plan.nodes.zero_()
        plan.replay()
        torch.cuda.synchronize()
        _cmp(plan.result(), exp, key_bits, (name, n, "graph"))
    short = gtc_mod.OctreePlan(ctx, n, key_bits, nodes_capacity=max(exp["n_oct_nodes"] - 1, 1))
    short.launch(d)
    assert short.counts_host()[2] == exp["n_oct_nodes"]
    assert ctx.device_status_code() == (7 if exp["n_oct_nodes"] > 1 else 0)


# Row kernels: 2..16 rows of 32 keys, 1..8 rows of 128 items per warp, 16 warps
# per block, one block per SM (two at the most rows); the sizes lie at a warp's,
# a block's and (for 152 SMs) each form's limit.
@pytest.mark.parametrize("n", [1, 2, 31, 33, 127, 129, 511, 513, 1023, 1024, 1025, 2048, 2049, 155_648, 155_649,
                               311_297, 622_593, 1_245_185, 2_490_369, 4_980_737])
@pytest.mark.parametrize("dups", [1, 40])
def test_row_scans(ctx, n, dups):
    """unique in place (both key widths, with and without values), the
    inclusive scan (aligned, unaligned, in place) and the node offsets, against
    numpy."""
    import torch

    g = np.random.Generator(np.random.PCG64(n + dups))
    for kd, td in ((np.uint32, np.int32), (np.uint64, np.int64)):
        keys = np.sort(g.integers(0, max(2 * n // dups, 2), n).astype(kd)) + kd(7)
        want, first = np.unique(keys, return_index=True)
        for with_vals in (True, False):
            k = torch.from_numpy(keys.view(td).copy()).cuda()
            v = torch.arange(n, dtype=torch.int32, device="cuda") if with_vals else None
            u = int(ctx.unique(k, v).item())
            assert u == want.size
            assert np.array_equal(k[:u].cpu().numpy().view(kd), want)
            if with_vals:
                assert np.array_equal(v[:u].cpu().numpy(), first)
    data = g.integers(0, 9, n + 8).astype(np.int32)
    d = torch.from_numpy(data).cuda()
    for lo in (0, 3, 4):
        assert np.array_equal(ctx.partial_sum(d, lo, lo + n).cpu().numpy(), np.cumsum(data[lo:lo + n], dtype=np.int32))
    e = torch.from_numpy(data[:n]).cuda()
    ps, o = ctx.node_offsets(e, n)
    want = np.concatenate((np.cumsum(data[:n], dtype=np.int32), [0]))
    want[n] = want[n - 1]
    want[0] = 0
    assert np.array_equal(ps.cpu().numpy(), want)
    assert int(o.item()) == 1 + want[n]
    L = ctx.L
    ctx.check(L.gtc_partial_sum_u32(ctx.h, d.data_ptr(), 0, n, d.data_ptr(), None, 0,
                                    torch.cuda.current_stream().cuda_stream))
    assert np.array_equal(d[:n].cpu().numpy(), np.cumsum(data[:n], dtype=np.int32))
    assert ctx.device_status() == 0


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("variant", [-1, 19, 20, 21])
def test_one_wave_sort(ctx, key_bits, variant):
    """The one-wave onesweep pass (default up to 175,000 or 200,000 keys, and pinned)
    and the shapes above it:
    tile edges, the untuned choice's crossings, the variants' own limits and
    one past them, narrow digits, unaligned inputs, the first-tile switch."""
    import torch

    kd, td = (np.uint32, np.int32) if key_bits == 32 else (np.uint64, np.int64)

    def check(keys, lo, hi, off=0):
        k = torch.from_numpy(keys.view(td).copy()).cuda()[off:]
        v = torch.arange(keys.size, dtype=torch.int32, device="cuda")[off:]
        want = keys[off:]
        digits = (want >> kd(lo)) & kd((1 << (hi - lo)) - 1)
        order = np.argsort(digits, kind="stable")
        for vals in (v, None):
            got = k.clone() if off == 0 else k
            ctx.sort_pairs(got, vals, lo, hi)
            assert np.array_equal(got.contiguous().cpu().numpy().view(kd), want[order]), (keys.size, lo, hi, off)
            if vals is not None:
                assert np.array_equal(vals.contiguous().cpu().numpy(), order.astype(np.int32) + off)
            if off:
                break

    try:
        ctx.set_sort_variant(key_bits, variant)
        for n in (1, 31, 255, 257, 1023, 1024, 1025, 4097, 78_000, 78_001, 163_840, 163_841, 175_000, 175_001, 200_000,
                  200_001, 409_600, 409_601, 622_592, 622_593, 1_245_185, 1_867_777):
            check(W.config3_keys(n, key_bits, and_words=n % 4, seed=n), 0, key_bits)
        for n in (5000, 120_007):
            keys = W.config3_keys(n, key_bits, seed=n)
            check(keys, 0, 30 if key_bits == 32 else 63)
            check(keys, 3, 8)
            check(keys, 0, key_bits, off=1)
            check(np.full(n, 7, kd), 0, key_bits)
        for db in (6, 7):
            ctx.set_sort_digit_bits(key_bits, db)
            check(W.config3_keys(70_001, key_bits, seed=db), 0, 40 if key_bits == 64 else 32)
        ctx.set_sort_digit_bits(key_bits, -1)
        assert ctx.device_status() == 0
        ctx.set_spin_limit(1000)
        ctx.debug_skip_first_tile()
        k = torch.from_numpy(W.config3_keys(20_000, key_bits, seed=3).view(td)).cuda()
        ctx.sort_pairs(k, None)
        assert ctx.device_status_code() == 4  # GTC_ERR_TIMEOUT
    finally:
        ctx.set_spin_limit(0)
        ctx.set_sort_digit_bits(key_bits, -1)
        ctx.set_sort_variant(key_bits, -1)
    check(W.config3_keys(20_000, key_bits, seed=3), 0, key_bits)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("side", ["right", "left", "both"])
def test_tree_nested_long_ranges(ctx, gtc_mod, key_bits, side):
    """Codes whose root paths nest one long range per bit: 700 codes hang off
    every level of a path to the first code, the last one, or a middle one, so
    the blocks at its end hold as many splits reaching past their window as
    there can be."""
    import torch

    kd = np.uint32 if key_bits == 32 else np.uint64
    bits = 30 if key_bits == 32 else 63
    g = np.random.Generator(np.random.PCG64(5))
    path = {"right": (1 << bits) - 1, "left": 0, "both": 0x2AAAAAAAAAAAAAAA & ((1 << bits) - 1)}[side]
    parts = [np.array([path], np.uint64)]
    for b in range(bits - 1, 9, -1):  # the subtree beside the path at bit b
        base = ((path >> b) ^ 1) << b
        parts.append(np.uint64(base) + g.choice(1 << min(b, 20), min(700, 1 << b), replace=False).astype(np.uint64))
    codes = np.unique(np.concatenate(parts)).astype(kd)
    d = torch.from_numpy(codes.view(np.int32 if key_bits == 32 else np.int64)).cuda()
    got = ctx.radix_tree(d, codes.size - 1, with_edge=True)
    try:
        gtc_mod.lib().gtc_tree_set_method(0)
        want = ctx.radix_tree(d, codes.size - 1, with_edge=True)
    finally:
        gtc_mod.lib().gtc_tree_set_method(1)
    for f in want:
        assert torch.equal(got[f], want[f]), f


def _spread_clouds(total, seed):
    """Clouds that add up to `total` points: empty ones first, last and in
    runs, single points, equal points across row and tile edges, and the rest
    split over a few large ones."""
    g = np.random.Generator(np.random.PCG64(seed))
    small = [0, 0, 1, 31, 0, 32, 33, 0, 0, 0, 1, 2047, 2048, 2049, 1, 1, 4097]
    big = total - sum(small)
    sizes = small + [big // 3, 0, big // 2, 0, big - big // 3 - big // 2, 0, 0]
    clouds = []
    for k, n in enumerate(sizes):
        p = W.uniform_points(n, seed=seed + k) if n else np.zeros((0, 4), np.float32)
        if n and k % 3 == 0:
            p = p[g.integers(0, max(n // 5, 1), n)]  # five points per code
        clouds.append(p)
    return clouds


@pytest.mark.parametrize("total,variant", [(155_649, -1), (233_472, -1), (466_945, -1), (599_999, -1), (600_000, 5), (600_001, 5), (600_001, -1), (700_001, -1),
                                           (800_001, -1), (1_000_001, -1), (1_245_185, -1), (1_999_999, -1),
                                           (2_000_000, -1), (2_700_001, 6), (13_001, 6), (13_001, -1)])
def test_batched_sizes(ctx, gtc_mod, oracle, total, variant):
    """Both sides of every size rule of the batch (tile shape, tree window,
    unique's rows or segments), over a range that is no power of two."""
    import torch

    from test_gpu_pipeline import _cmp

    clouds = _spread_clouds(total, seed=total)
    off = np.concatenate(([0], np.cumsum([c.shape[0] for c in clouds]))).astype(np.uint32)
    pts = np.ascontiguousarray(np.concatenate(clouds))
    try:
        gtc_mod.batched_set_variant(variant)
        res = gtc_mod.build_octree_batched(ctx, torch.from_numpy(pts).cuda(), torch.from_numpy(off.view(np.int32)).cuda(),
                                           min_coord=-3.0, rng=1100.0)
    finally:
        gtc_mod.batched_set_variant(-1)
    for c, r in enumerate(res):
        if clouds[c].shape[0] == 0:
            assert (r.n_unique, r.n_brt_nodes, r.n_oct_nodes) == (0, 0, 0)
            continue
        exp, _ = oracle.build_octree(clouds[c], 32, min_coord=-3.0, rng=1100.0, threads=8)
        _cmp(r, exp, 32, (total, c))


def _nested_cloud(key_bits, side, seed):
    """Points at the centres of the finest cells whose codes nest one long
    range per bit (test_tree_nested_long_ranges), in shuffled order: octree
    nodes of every span, most levels of the path far wider than a block."""
    axis, bits = (10, 30) if key_bits == 32 else (21, 63)
    g = np.random.Generator(np.random.PCG64(seed))
    path = {"right": (1 << bits) - 1, "left": 0, "both": 0x2AAAAAAAAAAAAAAA & ((1 << bits) - 1)}[side]
    parts = [np.array([path], np.uint64)]
    for b in range(bits - 1, 8, -1):
        base = ((path >> b) ^ 1) << b
        parts.append(np.uint64(base) + g.choice(1 << min(b, 20), min(300, 1 << b), replace=False).astype(np.uint64))
    codes = np.unique(np.concatenate(parts))
    pts = np.ones((codes.size, 4), np.float32)
    for a in range(3):
        q = np.zeros(codes.size, np.uint64)
        for b in range(axis):
            q |= ((codes >> np.uint64(3 * b + a)) & np.uint64(1)) << np.uint64(b)
        pts[:, a] = (q.astype(np.float64) + 0.5) * (1024.0 / (1 << axis))
    return pts[g.permutation(codes.size)]


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("side", ["right", "left", "both"])
def test_octree_window_far_owners(ctx, gtc_mod, oracle, key_bits, side):
    """Octree nodes assembled in a block's window and those gathered past it,
    in the single and the batched build, against the oracle."""
    import torch

    from test_gpu_pipeline import _cmp

    clouds = [_nested_cloud(key_bits, side, 1), W.uniform_points(5000, seed=2), _nested_cloud(key_bits, side, 3)]
    for c, pts in enumerate(clouds):
        exp, _ = oracle.build_octree(pts, key_bits, threads=8)
        _cmp(gtc_mod.build_octree(ctx, torch.from_numpy(pts).cuda(), key_bits), exp, key_bits, (side, c))
    if key_bits == 32:
        off = np.concatenate(([0], np.cumsum([c.shape[0] for c in clouds]))).astype(np.int32)
        res = gtc_mod.build_octree_batched(ctx, torch.from_numpy(np.concatenate(clouds)).cuda(),
                                           torch.from_numpy(off).cuda())
        for c, r in enumerate(res):
            exp, _ = oracle.build_octree(clouds[c], 32, threads=8)
            _cmp(r, exp, 32, (side, c, "batch"))


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("n", [1888, 1889, 4097, 5665, 9441, 50_001])
def test_octree_window_tiles(ctx, gtc_mod, oracle, key_bits, n):
    """Code counts around the octree window's tiles of 1,888 splits (four
    thousand points and more take the stage kernels; a capacity one short is
    flagged and the rest written)."""
    import torch

    from test_gpu_pipeline import _cmp

    pts = np.concatenate((W.gaussian_mixture_points(max(n, 4097), 4, 3.0, noise=0.3, seed=n)[:n],
                          np.repeat(W.uniform_points(1, seed=n), max(4097 - n, 0), axis=0)))
    d = torch.from_numpy(np.ascontiguousarray(pts)).cuda()
    exp, _ = oracle.build_octree(pts, key_bits)
    plan = gtc_mod.OctreePlan(ctx, pts.shape[0], key_bits, nodes_capacity=exp["n_oct_nodes"])
    plan.launch(d)
    _cmp(plan.result(), exp, key_bits, n)
    short = gtc_mod.OctreePlan(ctx, pts.shape[0], key_bits, nodes_capacity=exp["n_oct_nodes"] - 1)
    short.launch(d)
    assert ctx.device_status_code() == 7
    got = gtc_mod.nodes_to_numpy(short.nodes)
    same = (got.view(np.int32).reshape(-1, 16) == exp["nodes"][:-1].view(np.int32).reshape(-1, 16)).all(axis=1)
    assert same.sum() >= same.size - 21  # only nodes that share an owner with the one that did not fit


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 511, 512, 513, 1023, 1025, 3073, 4095, 4096, 4097])
def test_one_block_sort(ctx, key_bits, n):
    """One block up to 4,096 keys, the passes above: any bit range, with and
    without values, aligned and not, under capture."""
    import torch

    kd, td = (np.uint32, np.int32) if key_bits == 32 else (np.uint64, np.int64)
    for words, lo, hi in ((0, 0, key_bits), (2, 0, key_bits - 2), (0, 5, 9), (4, 0, 1), (1, key_bits - 17, key_bits)):
        keys = W.config3_keys(n + 1, key_bits, and_words=words, seed=n + words)
        keys[-1] = keys[0]
        for off in (0, 1):
            want = keys[off:off + n]
            order = np.argsort((want >> kd(lo)) & kd((1 << (hi - lo)) - 1), kind="stable")
            k = torch.from_numpy(keys.view(td).copy()).cuda()[off:off + n]
            v = torch.arange(n + 1, dtype=torch.int32, device="cuda")[off:off + n]
            ctx.sort_pairs(k, v, lo, hi)
            assert np.array_equal(k.contiguous().cpu().numpy().view(kd), want[order]), (lo, hi, off)
            assert np.array_equal(v.contiguous().cpu().numpy(), order.astype(np.int32) + off), (lo, hi, off)
            k = torch.from_numpy(keys.view(td).copy()).cuda()[off:off + n]
            ctx.sort_pairs(k, None, lo, hi)
            assert np.array_equal(k.contiguous().cpu().numpy().view(kd), want[order]), (lo, hi, off, "keys only")
    src = torch.from_numpy(keys[:n].view(td).copy()).cuda()
    k, alt, ws = src.clone(), torch.empty_like(src), ctx.workspace(1, n, key_bits)
    ctx.sort_pairs(k, None, ws=ws, keys_alt=alt)
    torch.cuda.synchronize()
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(s):
        g.capture_begin()
        ctx.sort_pairs(k, None, ws=ws, keys_alt=alt)
        g.capture_end()
    k.copy_(src)
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(k.cpu().numpy().view(kd), np.sort(keys[:n]))
    assert ctx.device_status() == 0
