"""Network rows of a group evaluated together: the same bits as a row at a time, at the edges
of the runs of 16 rows, of the weight tiles (32 columns, 256 outputs) and of the groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,counts", [
    ((3, 256, 256, 64), [1, 15, 16, 17, 0, 33, 300]),
    ((3, 48, 40, 8), [1300]),
    ((1, 33, 31, 1), [2, 0, 0, 1400, 5]),
    ((33, 257, 300, 65), [40, 31, 32]),
    ((5, 1, 1, 300), [31] * 40),
])
def test_grouped_rows_match_single_rows(sfh, shape, counts):
    torch = pytest.importorskip("torch")
    from sfhgpu._lib import load
    L, ctx = load(), sfh.default_context()
    rng = np.random.default_rng(sum(counts))
    i, h1, h2, o = shape
    n = h1 * i + h1 + h2 * h1 + h2 + o * h2 + o
    G = len(counts)
    group = rng.permutation(np.repeat(np.arange(G), counts)).astype(np.int32)
    bad = []
    if G > 1:  # rows of no group: NaN, and nothing else disturbed
        bad = rng.choice(group.size, 3, replace=False)
        group[bad] = [-1, G, 2**30]
    B = group.size
    assert B >= 2 * G
    P = torch.as_tensor(rng.normal(size=(G, n)).astype(np.float32) * 0.3, device="cuda")
    X = torch.as_tensor(rng.normal(size=(B, i)).astype(np.float32), device="cuda")
    dg = torch.as_tensor(group, device="cuda")
    Y = torch.zeros((B, o), dtype=torch.float32, device="cuda")
    R = torch.zeros((B, o), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    run = lambda g, x, gr, b, y: L.sfh_mlp_forward_rows(ctx.handle, *shape, P.data_ptr(), g, x, gr, b, y)
    assert run(G, X.data_ptr(), dg.data_ptr() if G > 1 else None, B, Y.data_ptr()) == 0
    g1 = max(G, 2)  # one row of two groups or more: the row-per-block kernel
    for r in range(B):
        assert run(g1, X[r:].data_ptr(), dg[r:].data_ptr(), 1, R[r:].data_ptr()) == 0
    ctx.synchronize()
    y, ref = Y.cpu().numpy(), R.cpu().numpy()
    assert np.isnan(y[bad]).all() if len(bad) else True
    np.testing.assert_array_equal(y, ref)
