"""bin_cmd at the edges of its integer comparisons: signed zeros, infinities, NaN, values on and
next to edges, uneven edges far from the mean step, point counts around a block's share and
grids on both sides of the shared-memory line.  Unit weights: the bins are exact, against
numpy's search of the same edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ref(x, y, ex, ey):
    kx, ky = np.searchsorted(ex, x, side="right") - 1, np.searchsorted(ey, y, side="right") - 1
    ok = (x >= ex[0]) & (x < ex[-1]) & (y >= ey[0]) & (y < ey[-1])
    h = np.zeros((ex.size - 1, ey.size - 1))
    np.add.at(h, (kx[ok], ky[ok]), 1.0)
    return h


@pytest.mark.parametrize("n", [1, 3, 1023, 1025, 70001])
@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 5), (96, 128), (97, 128)])
@pytest.mark.parametrize("kind", ["even", "uneven", "signed"])
def test_bin_edges(sfh, n, nx, ny, kind):
    rng = np.random.default_rng(n + nx * 10 + len(kind))
    if kind == "even":
        ex, ey = np.linspace(-1.0, 1.0, nx + 1), np.linspace(20.0, 28.0, ny + 1)
    elif kind == "uneven":
        ex = np.concatenate([[-3.0], np.sort(rng.uniform(0.0, 1e-3, nx - 1)), [50.0]])
        ey = np.cumsum(rng.uniform(1e-6, 3.0, ny + 1))
    else:
        ex, ey = np.linspace(-5.0, 0.0, nx + 1), np.linspace(0.0, 1e-300, ny + 1)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, -np.nan, 5e-324, -5e-324])

    def draw(e):
        v = rng.uniform(e[0] - 0.01 * (e[-1] - e[0]), e[-1] * 1.0 + 0.01 * (e[-1] - e[0]), n)
        k = rng.integers(0, 4, n)
        on = e[rng.integers(0, e.size, n)]
        v = np.where(k == 0, on, np.where(k == 1, np.nextafter(on, -np.inf), v))
        pick = rng.random(n) < 0.05
        v[pick] = special[rng.integers(0, special.size, pick.sum())]
        return v
    x, y = draw(ex), draw(ey)
    H = sfh.bin_cmd(x, y, edges=(ex, ey)).weights
    with np.errstate(invalid="ignore"):
        assert np.array_equal(H, _ref(x, y, ex, ey))
