"""Stamps of wide stars (register tiles) and narrow stars (per-bin) against the FP64 oracle, at
the sizes where the tiling and the class line can go wrong.

Tolerance, from the error budget of the kernels: per bin 1e-5 |ref| + 1e-6 max(ref), that of
the template tests.  The wide form's own error is below 4e-7 of a bin's value down to 1e-4 of
the peak and 2e-8 of the peak below that; FP32 exponents of up to 2^-100 add about 1e-6 of a
bin's value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stars(rng, n, smin, smax, ratio):
    x = rng.uniform(-1.2, 3.0, n)
    y = rng.uniform(17.0, 33.0, n)
    sx = np.exp(rng.uniform(np.log(smin), np.log(smax), n))
    return x, y, sx, sx * np.exp(rng.uniform(-np.log(ratio), np.log(ratio), n)), rng.random(n) + 0.1


def _check(H, R):
    bound = 1e-5 * np.abs(R) + 1e-6 * np.abs(R).max()
    assert np.max(np.abs(H - R) / np.maximum(bound, 1e-300)) <= 1.0


def _ref(O, x, y, sx, sy, w, cov, xe, ye):
    nx, ny = xe.size - 1, ye.size - 1
    return O.bin_cmd_smooth(x, y, sx, sy, w, cov, (xe[0], (xe[-1] - xe[0]) / nx, nx),
                            (ye[0], (ye[-1] - ye[0]) / ny, ny))


@pytest.mark.parametrize("cov", [0, 1, -1])
@pytest.mark.parametrize("smin,smax,ratio", [(0.02, 0.6, 1.5), (0.3, 3.0, 1.2), (1.0, 600.0, 4.0),
                                             (0.05, 5.0, 60.0)])
@pytest.mark.parametrize("nx,ny,n", [(2, 2, 40), (8, 8, 40), (7, 9, 40), (64, 33, 300),
                                     (65, 129, 257), (257, 40, 300), (200, 300, 700)])
def test_stamp_classes(sfh, O, cov, smin, smax, ratio, nx, ny, n):
    rng = np.random.default_rng(nx * 1000 + ny + n + int(10 * smax) + cov)
    xe, ye = np.linspace(-0.6, 2.4, nx + 1), np.linspace(19.0, 30.0, ny + 1)
    x, y, sx, sy, w = _stars(rng, n, smin, smax, ratio)
    H = sfh.bin_cmd_smooth(x, y, sx, sy, cov, weights=w, edges=(xe, ye)).weights
    _check(H, _ref(O, x, y, sx, sy, w, cov, xe, ye))


@pytest.mark.parametrize("nx,ny", [(3100, 5), (2057, 17), (3, 2100)])
def test_stamp_extreme_grids(sfh, O, nx, ny):
    """The widest accepted grid (several passes of tiles per band) and a tall narrow one."""
    rng = np.random.default_rng(nx)
    xe, ye = np.linspace(-0.6, 2.4, nx + 1), np.linspace(19.0, 30.0, ny + 1)
    x, y, sx, sy, w = _stars(rng, 60, 0.02, 20.0, 1.5)
    for cov in (0, 1):
        H = sfh.bin_cmd_smooth(x, y, sx, sy, cov, weights=w, edges=(xe, ye)).weights
        _check(H, _ref(O, x, y, sx, sy, w, cov, xe, ye))


@pytest.mark.parametrize("cov", [0, 1])
def test_stamps_with_device_offsets(sfh, O, cov):
    """sfh_bin_cmd_smooth_batch_dev: star counts known on the device only."""
    import torch
    from sfhgpu._lib import check, load
    rng = np.random.default_rng(5)
    nx, ny, counts = 61, 47, [0, 1, 255, 300]
    xe, ye = np.linspace(-0.6, 2.4, nx + 1), np.linspace(19.0, 30.0, ny + 1)
    st = [_stars(rng, n, 0.03, 30.0, 1.5) for n in counts]
    dev = torch.device("cuda", 0)
    cols = [torch.as_tensor(np.concatenate([s[k] for s in st]), device=dev) for k in range(5)]
    off = torch.as_tensor(np.concatenate([[0], np.cumsum(counts)]).astype(np.int64), device=dev)
    out = torch.empty((len(counts), ny * nx), dtype=torch.float32, device=dev)
    hcov = np.full(len(counts), cov, dtype=np.int32)
    ctx = sfh.default_context()
    torch.cuda.synchronize()
    check(load().sfh_bin_cmd_smooth_batch_dev(
        ctx.handle, *[c.data_ptr() for c in cols], off.data_ptr(), hcov.ctypes.data, len(counts),
        float(xe[0]), float((xe[-1] - xe[0]) / nx), nx, float(ye[0]),
        float((ye[-1] - ye[0]) / ny), ny, out.data_ptr()), ctx.handle, "batch_dev")
    ctx.synchronize()
    for t, s in enumerate(st):
        G = out[t].cpu().numpy().reshape(ny, nx).T
        if counts[t] == 0:
            assert not G.any()
        else:
            _check(G, _ref(O, *s, cov, xe, ye))


def test_non_finite_weight_stays_in_its_window(sfh):
    """A star with an infinite weight changes only the bins of its own window."""
    xe, ye = np.linspace(0.0, 4.0, 201), np.linspace(0.0, 4.0, 201)
    x, y, s = np.array([1.0, 2.0]), np.array([1.0, 2.0]), np.array([0.3, 0.3])
    H = sfh.bin_cmd_smooth(x, y, s, s, 0, weights=np.array([np.inf, 1.0]), edges=(xe, ye)).weights
    xo = int(np.ceil(10 * 0.3 / 0.02)) // 2
    cx = int(np.rint(1.0 / 0.02 + 1.0)) - 1
    assert np.isfinite(H[cx + xo + 1:, :]).all() and np.isfinite(H[:, cx + xo + 1:]).all()
    assert not np.isfinite(H[cx, cx])
