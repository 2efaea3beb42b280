"""Network rows spread unevenly over the groups: the same bits as a row at a time, and no group
that holds most of the rows left to a few blocks."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPE = (3, 256, 256, 64)


def _inputs(G, group):
    import torch
    i, h1, h2, o = SHAPE
    n = h1 * i + h1 + h2 * h1 + h2 + o * h2 + o
    g = torch.Generator(device="cuda").manual_seed(G)
    P = 0.1 * torch.randn((G, n), generator=g, device="cuda")
    X = torch.randn((group.size, i), generator=g, device="cuda")
    return P, X, torch.as_tensor(group.astype(np.int32), device="cuda")


@pytest.mark.parametrize("G,B,share", [(64, 1200, 1.0), (64, 1200, 0.5), (300, 700, 0.9), (8448, 16900, 0.02),
                                       (8449, 16900, 0.02)])
def test_uneven_groups_match_single_rows(sfh, G, B, share):
    """`share` of the rows in the last group, the others anywhere, some in no group."""
    import torch
    from sfhgpu._lib import load
    L, ctx = load(), sfh.default_context()
    rng = np.random.default_rng(G + B)
    group = np.where(rng.random(B) < share, G - 1, rng.integers(0, G, B))
    group[rng.choice(B, 3, replace=False)] = [-1, G, -2**31]
    P, X, dg = _inputs(G, group)
    Y = torch.zeros((B, SHAPE[3]), device="cuda")
    R = torch.zeros_like(Y)
    torch.cuda.synchronize()
    assert L.sfh_mlp_forward_rows(ctx.handle, *SHAPE, P.data_ptr(), G, X.data_ptr(), dg.data_ptr(), B,
                                  Y.data_ptr()) == 0
    some = np.unique(np.concatenate([rng.choice(B, 200), np.flatnonzero((group < 0) | (group >= G)),
                                     [0, B - 1]]))
    for r in some:  # one row of two groups or more: the row-per-block kernel
        assert L.sfh_mlp_forward_rows(ctx.handle, *SHAPE, P.data_ptr(), G, X[r:].data_ptr(),
                                      dg[r:].data_ptr(), 1, R[r:].data_ptr()) == 0
    ctx.synchronize()
    y, ref = Y.cpu().numpy()[some], R.cpu().numpy()[some]
    np.testing.assert_array_equal(y, ref)
    bad = (group[some] < 0) | (group[some] >= G)
    assert np.isnan(y[bad]).all() and np.isfinite(y[~bad]).all()


@pytest.mark.parametrize("G,B", [(64, 10000), (512, 2048)])
def test_one_group_takes_about_as_long_as_many(sfh, G, B):
    """All rows in one group: a few times the even spread at most (its weights are read fewer times,
    its rows are as many); a group left to its mean number of blocks takes 15 to 40 times as long."""
    import torch
    from sfhgpu._lib import load
    L, ctx = load(), sfh.default_context()
    took = []
    for group in (np.arange(B) % G, np.zeros(B)):
        P, X, dg = _inputs(G, group)
        Y = torch.empty((B, SHAPE[3]), device="cuda")
        torch.cuda.synchronize()
        best = np.inf
        for _ in range(8):
            t = time.perf_counter()
            assert L.sfh_mlp_forward_rows(ctx.handle, *SHAPE, P.data_ptr(), G, X.data_ptr(),
                                          dg.data_ptr(), B, Y.data_ptr()) == 0
            ctx.synchronize()
            best = min(best, time.perf_counter() - t)
        took.append(best)
    assert took[1] < 5 * took[0], took
