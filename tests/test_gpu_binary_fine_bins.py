"""binary_hess on bins finer than the FP32 logarithm of a pair's magnitudes (2e-9): a pair in the first or
last bin of such an axis is binned from its FP64 magnitudes, as on any other.

Tolerance as for the other binary templates: per bin 1e-4 relative + 1e-5 of the maximum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_pairs_in_the_outer_bins_of_fine_axes(sfh, O):
    torch = pytest.importorskip("torch")
    from sfhgpu import synthetic as S
    dev = torch.device("cuda", 0)
    E = [O.ErrModel(e.a, e.b, e.c, e.d, e.cap) for e in S.error_models()]
    Cm = [O.ComplModel(c.A, c.m50, c.rho) for c in S.completeness_models()]
    imf, nx, ny, seen = O.kroupa2001(), 6, 5, 0
    rng = np.random.default_rng(8)
    for trial in range(60):
        # three points: two intervals, one pair
        m = np.sort(rng.uniform(0.3, 1.2, 3))
        mags = np.ascontiguousarray(rng.uniform(22.0, 26.0, (3, 3)))
        f = 10.0 ** (-0.4 * mags[:, :2])
        b, v = -2.5 * np.log10(f[:2].sum(axis=1))
        xs = ys = 2.0**-35  # 2.9e-11
        # the pair in the middle of the first or the last bin of each axis
        ix, iy = rng.choice([0, nx - 1]), rng.choice([0, ny - 1])
        xf, yf = (b - v) - (ix + 0.5) * xs, v - (iy + 0.5) * ys
        xe, ye = xf + xs * np.arange(nx + 1), yf + ys * np.arange(ny + 1)
        gx, gy = (xe[0], (xe[-1] - xe[0]) / nx, nx), (ye[0], (ye[-1] - ye[0]) / ny, ny)
        ref = O.binary_hess(m, mags, E, Cm, 1, (0, 1), imf, 1.0, O.imf_mean(imf), gx, gy)
        seen += ref.sum() > 0
        got = sfh.binary_hess_batch(
            torch.tensor(m, device=dev), torch.tensor(mags, device=dev), [0], [3], 1, (0, 1),
            S.error_models(), S.completeness_models(), S.imf(), 1.0,
            (sfh.Range(list(xe), gx[1]), sfh.Range(list(ye), gy[1])))
        got = got.cpu().numpy()[0].reshape(ny, nx).T
        assert np.all(np.abs(got - ref) <= 1e-4 * np.abs(ref) + 1e-5 * np.abs(ref).max()), trial
    assert seen > 40
