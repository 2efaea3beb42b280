"""fg! on FP64 templates takes one launch only where that is the faster form (four kernels are faster
from 128 templates on with more 64-bin tiles than SMs, and for most matrices of more than 256)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,tiles,launches", [
    (1, 1, 1), (50, 118, 1), (20, 304, 1), (20, 305, 4), (96, 304, 1), (120, 240, 1), (127, 304, 4),
    (128, 152, 1), (128, 153, 4), (160, 228, 4), (199, 304, 4), (255, 152, 1), (255, 153, 4),
    (256, 59, 1), (256, 60, 4), (256, 152, 4), (400, 38, 1), (400, 152, 4), (408, 10, 4)])
def test_route_of_fp64_fg(sfh, O, nt, tiles, launches):
    nb = 64 * tiles - 5
    rng = np.random.default_rng(nt + tiles)
    M = np.asfortranarray(rng.random((nb, nt)))
    r = rng.random(nt)
    data = rng.poisson(M @ r).astype(float)
    H = sfh.Models(M, storage="f64")
    G, comp = np.empty(nt), np.empty(nb)
    sfh.fg_(True, G, r, H, data, comp)
    before = H.ctx.launches
    v = sfh.fg_(True, G, r, H, data, comp)
    assert H.ctx.launches - before == launches
    v_ref, G_ref, _ = O.fg(r, M, data)
    # FP64 sums of at most 2e4 terms
    c = M @ r
    assert abs(v - v_ref) <= 1e-10 * (np.abs(data - c) + data * np.abs(np.log(np.maximum(data, 1) / c))).sum()
    assert np.all(np.abs(G - G_ref) <= 1e-10 * (np.abs(M).T @ np.abs(1 - data / c)))
