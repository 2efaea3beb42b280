"""sfh_bin_cmd_smooth_batch_dev (star counts known on the device only): narrow, mid and wide stars at
counts around a warp's share, on grids whose rows are written by 16 bytes and by 4; many templates of
narrow stars cost a fraction of a microsecond each.

Tolerance, that of the template tests: per bin 1e-5 |ref| + 1e-6 max(ref)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(sfh, cols, counts, cov, nx, ny, xf, xs, yf, ys, repeat=1):
    import torch
    from sfhgpu._lib import check, load
    dev, ctx = torch.device("cuda", 0), sfh.default_context()
    d = [torch.as_tensor(c, device=dev) for c in cols]
    off = torch.as_tensor(np.concatenate([[0], np.cumsum(counts)]).astype(np.int64), device=dev)
    out = torch.full((len(counts), ny * nx), np.nan, dtype=torch.float32, device=dev)
    hcov = np.full(len(counts), cov, dtype=np.int32)
    torch.cuda.synchronize()
    best = np.inf
    for _ in range(repeat):
        t = time.perf_counter()
        check(load().sfh_bin_cmd_smooth_batch_dev(
            ctx.handle, *[c.data_ptr() for c in d], off.data_ptr(), hcov.ctypes.data, len(counts), xf,
            xs, nx, yf, ys, ny, out.data_ptr()), ctx.handle, "batch_dev")
        ctx.synchronize()
        best = min(best, time.perf_counter() - t)
    return out.cpu().numpy().reshape(len(counts), ny, nx).transpose(0, 2, 1), best


@pytest.mark.parametrize("cov", [0, 1, -1])
@pytest.mark.parametrize("nx,ny", [(100, 50), (102, 33), (7, 9), (64, 64)])
@pytest.mark.parametrize("ntempl", [1, 40, 1500])
def test_device_counts(sfh, O, cov, nx, ny, ntempl):
    rng = np.random.default_rng(nx + ntempl + cov)
    counts = rng.choice([0, 1, 2, 9, 31, 32, 33, 65], ntempl)
    counts[0] = 257
    n = int(counts.sum())
    xs, ys = 3.0 / nx, 11.0 / ny
    x, y, w = rng.uniform(-0.9, 2.7, n), rng.uniform(18.0, 31.0, n), rng.random(n) + 0.1
    sx = xs * np.exp(rng.uniform(np.log(0.05), np.log(60.0), n))
    sy = sx * (ys / xs) * np.exp(rng.uniform(-0.5, 0.5, n))
    got, _ = _run(sfh, (x, y, sx, sy, w), counts, cov, nx, ny, -0.6, xs, 19.0, ys)
    off = np.concatenate([[0], np.cumsum(counts)])
    for t in {0, ntempl - 1, *rng.choice(ntempl, min(ntempl, 25)).tolist()}:
        sl = slice(off[t], off[t + 1])
        if counts[t] == 0:
            assert not got[t].any()
            continue
        R = O.bin_cmd_smooth(x[sl], y[sl], sx[sl], sy[sl], w[sl], cov, (-0.6, xs, nx), (19.0, ys, ny))
        assert np.all(np.abs(got[t] - R) <= 1e-5 * np.abs(R) + 1e-6 * np.abs(R).max())


def test_narrow_stars_of_many_templates(sfh):
    """3,000 templates of 100 narrow stars against the same templates of one: a hundred times the
    stars, and less than five times the time (nearly nine with a record per warp)."""
    rng = np.random.default_rng(1)
    took = []
    for per in (1, 100):
        n = 3000 * per
        s = np.full(n, 0.2)
        cols = (rng.random(n), rng.random(n), s / 100, s / 150, np.ones(n))
        took.append(_run(sfh, cols, [per] * 3000, 0, 100, 150, 0.0, 0.01, 0.0, 1 / 150, 8)[1])
    assert took[1] < 5 * took[0], took
