"""bin_cmd_smooth of a few stars: no launch for Chebyshev tiles below 64 stars, and the oracle's
template on both sides of that line and of the warps per tile group.

Tolerance, that of the template tests: per bin 1e-5 |ref| + 1e-6 max(ref)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cov", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 17, 63, 64, 65])
def test_few_stars(sfh, O, cov, n):
    rng = np.random.default_rng(n)
    nx, ny = 200, 300
    xe, ye = np.linspace(-0.6, 2.4, nx + 1), np.linspace(19.0, 30.0, ny + 1)
    x, y, w = rng.uniform(0.0, 2.0, n), rng.uniform(20.0, 29.0, n), rng.random(n) + 0.1
    sx = np.exp(rng.uniform(np.log(0.005), np.log(30.0), n))
    sy = sx * rng.uniform(0.8, 1.2, n)
    ctx = sfh.default_context()
    before = ctx.launches
    H = sfh.bin_cmd_smooth(x, y, sx, sy, cov, weights=w, edges=(xe, ye), ctx=ctx).weights
    assert ctx.launches - before == (3 if n < 64 else 4)
    R = O.bin_cmd_smooth(x, y, sx, sy, w, cov, (xe[0], (xe[-1] - xe[0]) / nx, nx),
                         (ye[0], (ye[-1] - ye[0]) / ny, ny))
    assert np.all(np.abs(H - R) <= 1e-5 * np.abs(R) + 1e-6 * np.abs(R).max())
