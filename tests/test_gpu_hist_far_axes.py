"""bin_cmd on axes whose offset is large against their step: the bins are numpy's, and a point costs
what it costs near zero (guesses from values rounded to FP32 start hundreds of bins away)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first,width,nx", [(2.45e6, 3.0, 300), (2.45e6, 0.2, 4000), (1e5, 1.0, 300),
                                            (-1e9, 10.0, 2000), (3e300, 1e300, 500), (-2.0, 1e-9, 700),
                                            (1e15, 4096.0, 4096), (0.0, 1.0, 200)])
@pytest.mark.parametrize("n", [1, 1023, 60001])
def test_far_axes(sfh, first, width, nx, n):
    rng = np.random.default_rng(n + nx)
    ex, ey = np.linspace(first, first + width, nx + 1), np.linspace(20.0, 28.0, 11)
    x, y = rng.uniform(ex[0], ex[-1], n), rng.uniform(19.5, 28.5, n)
    on = rng.random(n) < 0.3
    x[on] = ex[rng.integers(0, ex.size, on.sum())]
    x = np.where(rng.random(n) < 0.2, np.nextafter(x, -np.inf), x)
    H = sfh.bin_cmd(x, y, edges=(ex, ey)).weights
    kx, ky = np.searchsorted(ex, x, side="right") - 1, np.searchsorted(ey, y, side="right") - 1
    ok = (x >= ex[0]) & (x < ex[-1]) & (y >= ey[0]) & (y < ey[-1])
    ref = np.zeros((nx, 10))
    np.add.at(ref, (kx[ok], ky[ok]), 1.0)
    assert np.array_equal(H, ref)


def test_far_axis_takes_as_long_as_a_near_one(sfh):
    import torch
    from sfhgpu._lib import load
    L, ctx, dev = load(), sfh.default_context(), torch.device("cuda", 0)
    n, nx, ny, took = 500000, 4000, 100, []
    rng = np.random.default_rng(4)
    for first in (0.0, 2.45e6):
        ex, ey = np.linspace(first, first + 0.2, nx + 1), np.linspace(20.0, 28.0, ny + 1)
        d = [torch.as_tensor(v, device=dev) for v in
             (rng.uniform(ex[0], ex[-1], n), rng.uniform(20.0, 28.0, n), ex, ey)]
        out = torch.empty(nx * ny, dtype=torch.float64, device=dev)
        torch.cuda.synchronize()
        best = np.inf
        for _ in range(10):
            t = time.perf_counter()
            assert L.sfh_bin_cmd_dev(ctx.handle, d[0].data_ptr(), d[1].data_ptr(), None, n,
                                     d[2].data_ptr(), nx, d[3].data_ptr(), ny, out.data_ptr()) == 0
            ctx.synchronize()
            best = min(best, time.perf_counter() - t)
        took.append(best)
    assert took[1] < 5 * took[0], took
