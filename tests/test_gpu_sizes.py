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
@pytest.mark.parametrize("u", [2, 1023, 1024, 1025, 1026, 2049, 4096, 4097, 9000, 700_000, 700_001, 700_002, 708_609])
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
