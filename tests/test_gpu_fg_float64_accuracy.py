"""G of fg! on FP64 templates against extended precision, where a thread of the one-launch form sums a
tile's 64 bins alone (128 to 255 templates).

Tolerance: an emulation of the sums in numpy on these inputs gives a mean error of 3.3e-16 (norm of
the error over norm of G) for four sums of 16 bins and 9.6e-16 to 1.2e-15 for one sum of 64; w itself
is known to about 1.5e-16.  The bound is 7.5e-16."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(nt, nx, ny, seed):
    """Hess-diagram templates of stars of growing error, coefficients around those of the counts."""
    import torch
    g = torch.Generator().manual_seed(seed)
    u = torch.rand((nt, 64), generator=g, dtype=torch.float64)
    age = torch.linspace(0, 1, nt, dtype=torch.float64)[:, None]
    y = 2.0 * age + (10.0 - 2.0 * age) * u
    x = 0.9 + 0.5 * (u - 0.4 - 0.3 * age) ** 2 + 0.15 * age
    s = 0.01 + 0.15 * torch.exp((y - 8.5) / 1.2)
    w = torch.exp(1.2 * (y - 6.5) / 2.5) / (1.0 + torch.exp((y - 8.5) / 0.3))

    def part(c, hi, n, sc):
        e = torch.linspace(0, hi, n + 1, dtype=torch.float64)
        t = torch.special.erf((e[None, None, :] - c[:, :, None]) / (2.0**0.5 * sc[:, :, None]))
        return t[:, :, 1:] - t[:, :, :-1]
    M = torch.bmm((part(y, 11.0, ny, s) * w[:, :, None]).transpose(1, 2), part(x, 3.0, nx, 1.4 * s))
    M = M.reshape(nt, ny * nx).numpy() + 1e-9
    rng = np.random.default_rng(seed)
    r = np.exp(rng.standard_normal(nt))
    r *= 2e4 / (r @ M).sum()
    return M, r * np.exp(0.2 * rng.standard_normal(nt)), rng.poisson(r @ M).astype(float)


@pytest.mark.parametrize("nt,nx,ny", [(129, 52, 147), (171, 48, 52), (255, 60, 100)])
def test_gradient_in_extended_precision(sfh, nt, nx, ny):
    L, off = np.longdouble, []
    for seed in range(8):
        M, r, data = _inputs(nt, nx, ny, seed)
        H = sfh.Models(np.asfortranarray(M.T), storage="f64")
        G, comp = np.empty(nt), np.empty(nx * ny)
        sfh.fg_(True, G, r, H, data, comp)
        Me = M.astype(L)
        ref = Me @ (1 - data / (r.astype(L) @ Me))
        off.append(float(np.sqrt(((G - ref) ** 2).sum() / (ref**2).sum())))
    assert np.mean(off) < 7.5e-16, off
