"""The C entry points of the template builds refuse grids out of range with an error code."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,name", [
    (0, 10, "ARG"), (10, 0, "ARG"), (-40, 10, "ARG"), (10, -40, "ARG"), (5 - 2**32, 10, "ARG"),
    ((1 << 20) + 1, 10, "ARG"), (10, (1 << 20) + 1, "ARG"), (3124, 10, "UNSUPPORTED")])
def test_grids_out_of_range(sfh, nx, ny, name):
    import torch
    from sfhgpu import _lib
    from sfhgpu import synthetic as S
    from sfhgpu.templates import ComplModel, ErrModel
    want = getattr(_lib, "SFH_ERR_" + name)
    L, ctx, dev = _lib.load(), sfh.default_context(), torch.device("cuda", 0)
    m, mags = S.isochrone(9.0, -1.0, 50)
    d_m, d_mags = torch.tensor(m, device=dev), torch.tensor(mags, device=dev)
    out = torch.zeros(64, dtype=torch.float32, device=dev)
    off, ln = np.zeros(1, dtype=np.int64), np.array([50], dtype=np.int32)
    one, dm = np.ones(1), np.array([25.0])
    E, K = (ErrModel * 3)(*S.error_models()), (ComplModel * 3)(*S.completeness_models())
    imf = S.imf()
    ip = imf.params()
    torch.cuda.synchronize()
    assert L.sfh_partial_cmd_smooth_batch_dev(
        ctx.handle, d_m.data_ptr(), d_mags.data_ptr(), 50, off.ctypes.data, ln.ctypes.data, 1, 3, 1,
        0, 1, E, K, None, C.byref(ip), imf.mean(), dm.ctypes.data, one.ctypes.data, -0.6, 0.3, nx,
        19.0, 1.1, ny, out.data_ptr()) == want
    star = torch.ones(4, dtype=torch.float64, device=dev)
    offs = torch.tensor([0, 4], dtype=torch.int64, device=dev)
    cov = np.ones(1, dtype=np.int32)
    torch.cuda.synchronize()
    assert L.sfh_bin_cmd_smooth_batch_dev(
        ctx.handle, *[star.data_ptr()] * 5, offs.data_ptr(), cov.ctypes.data, 1, -0.6, 0.3, nx, 19.0,
        1.1, ny, out.data_ptr()) == want
    ctx.synchronize()
    assert not out.cpu().numpy().any()


@pytest.mark.parametrize("npts", [216, 300, 500])
def test_more_resampled_points_than_an_int_counts(sfh, npts):
    """Bins so fine that a template's resampled points pass 2^31 (and, wrapped, come out negative or
    small again): refused, and the next call is served."""
    import torch
    from sfhgpu import _lib
    from sfhgpu import synthetic as S
    dev = torch.device("cuda", 0)
    m, mags = S.isochrone(9.0, -1.0, npts)

    def build(step):
        xe, ye = 0.5 + step * np.arange(11), 25.0 + step * np.arange(11)
        return sfh.partial_cmd_smooth_batch(
            torch.tensor(np.concatenate([m, m]), device=dev),
            torch.tensor(np.concatenate([mags, mags], axis=1), device=dev), [0, npts], [npts, npts],
            1, (0, 1), S.error_models(), S.completeness_models(), S.imf(), 25.0, 1.0, (xe, ye))
    with pytest.raises(_lib.SFHError) as e:
        build(2.0**-40)
    assert e.value.status == _lib.SFH_ERR_NOMEM
    assert np.isfinite(build(0.25).cpu().numpy()).all()
