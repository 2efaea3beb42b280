"""Stars whose two errors differ by many orders of magnitude and descending bin edges, against the
FP64 oracle.

Tolerance, that of the template tests: per bin 1e-5 |ref| + 1e-6 max(ref)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(sfh, O, x, y, sx, sy, cov, xe, ye):
    x, y, sx, sy = (np.atleast_1d(np.asarray(v, dtype=float)) for v in np.broadcast_arrays(x, y, sx, sy))
    w = np.linspace(0.5, 1.5, x.size)
    H = sfh.bin_cmd_smooth(x, y, sx, sy, cov, weights=w, edges=(xe, ye)).weights
    nx, ny = xe.size - 1, ye.size - 1
    R = O.bin_cmd_smooth(x, y, sx, sy, w, cov, (xe[0], (xe[-1] - xe[0]) / nx, nx),
                         (ye[0], (ye[-1] - ye[0]) / ny, ny))
    assert np.isfinite(H).all() and np.abs(R).max() > 0
    assert np.all(np.abs(H - R) <= 1e-5 * np.abs(R) + 1e-6 * np.abs(R).max())


@pytest.mark.parametrize("cov", [1, -1])
@pytest.mark.parametrize("sy", [1e2, 1e4, 1e5, 1e6])
def test_wide_star_with_a_far_larger_y_error(sfh, O, cov, sy):
    xe, ye = np.linspace(-0.6, 2.4, 201), np.linspace(19.0, 30.0, 301)
    _check(sfh, O, [0.4, 0.9, 1.3], [24.0, 25.1, 27.3], [0.4, 0.5, 0.7], [sy, 1.3 * sy, 1.7 * sy],
           cov, xe, ye)


@pytest.mark.parametrize("cov", [1, -1])
@pytest.mark.parametrize("flip", [(True, False), (False, True), (True, True)])
def test_descending_edges(sfh, O, cov, flip):
    """A negative bin step of a covariant star: the window of three bins and the integrals of the
    opposite sign that the reference's formulas give."""
    rng = np.random.default_rng(3)
    n, nx, ny = 40, 30, 25
    xe, ye = np.linspace(-0.6, 2.4, nx + 1), np.linspace(19.0, 30.0, ny + 1)
    xe, ye = xe[::-1].copy() if flip[0] else xe, ye[::-1].copy() if flip[1] else ye
    x, y, w = rng.uniform(-0.5, 2.3, n), rng.uniform(19.5, 29.5, n), rng.random(n) + 0.1
    sx, sy = rng.uniform(0.5, 1.5, n), rng.uniform(2.0, 6.0, n)
    H = sfh.bin_cmd_smooth(x, y, sx, sy, cov, weights=w, edges=(xe, ye)).weights
    R = O.bin_cmd_smooth(x, y, sx, sy, w, cov, (xe[0], (xe[-1] - xe[0]) / nx, nx),
                         (ye[0], (ye[-1] - ye[0]) / ny, ny))
    assert np.all(np.abs(H - R) <= 1e-5 * np.abs(R) + 1e-6 * np.abs(R).max())


@pytest.mark.parametrize("cov", [1, -1])
@pytest.mark.parametrize("nx,ny,xs,ys", [(277, 6, 0.0034, 1.6), (92, 20, 0.007, 1.8), (74, 6, 0.008, 6.1)])
def test_y_steps_of_thousands_of_x_errors(sfh, O, cov, nx, ny, xs, ys):
    """Stars of a few bins or less in x whose shear over one row is up to 1e5 x errors."""
    rng = np.random.default_rng(nx + cov)
    xe, ye = 0.1 + xs * np.arange(nx + 1), 20.0 + ys * np.arange(ny + 1)
    n = 400
    sx = xs * np.exp(rng.uniform(np.log(0.01), np.log(5.0), n))
    sy = np.where(rng.random(n) < 0.5, sx * ys / xs, ys * np.exp(rng.uniform(np.log(0.002), np.log(3.0), n)))
    _check(sfh, O, rng.uniform(xe[0], xe[-1], n), rng.uniform(ye[0], ye[-1], n), sx, sy, cov, xe, ye)
