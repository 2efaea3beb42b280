"""binary_hess on grids whose bins are coarse, fine or unlike on the two axes: pairs binned from an
FP32 position and, near a bin's edge, from FP64 logarithms fall where the FP64 oracle puts them.

Tolerance as for the other binary templates: per bin 1e-4 relative + 1e-5 of the maximum; a pair on
the wrong side of an edge moves whole pairs' weights, far more than that on the coarse grids."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,y_index", [(3, 4, 1), (2, 300, 0), (200, 3, 1), (64, 65, 0)])
def test_pairs_fall_into_the_oracles_bins(sfh, O, nx, ny, y_index):
    torch = pytest.importorskip("torch")
    from sfhgpu import synthetic as S
    E = [O.ErrModel(e.a, e.b, e.c, e.d, e.cap) for e in S.error_models()]
    Cm = [O.ComplModel(c.A, c.m50, c.rho) for c in S.completeness_models()]
    w = S.small(nages=1, nmh=2)
    m_ini, mags, offs, lens = S.isochrone_batch(w)
    mags = np.ascontiguousarray(mags + 1e-6 * np.random.default_rng(nx).random(mags.shape))
    ex = np.linspace(w.xedges[0], w.xedges[-1], nx + 1)
    ey = np.linspace(w.yedges[0], w.yedges[-1], ny + 1)
    pts = [sfh.binary_points(m_ini[o:o + n], list(mags[:, o:o + n]), y_index, (0, 1), w.dmod,
                             (w.xedges, w.yedges)) for o, n in zip(offs, lens)]
    ln = np.array([p[0].size for p in pts], dtype=np.int32)
    of = np.concatenate([[0], np.cumsum(ln)[:-1]]).astype(np.int64)
    dev = torch.device("cuda", 0)
    out = sfh.binary_hess_batch(torch.tensor(np.concatenate([p[0] for p in pts]), device=dev),
                                torch.tensor(np.concatenate([p[1] for p in pts], axis=1), device=dev),
                                of, ln, y_index, (0, 1), S.error_models(), S.completeness_models(),
                                S.imf(), w.normalize_value, (ex, ey))
    torch.cuda.synchronize()
    out = out.cpu().numpy()
    imf = O.kroupa2001()
    gx, gy = (ex[0], (ex[-1] - ex[0]) / nx, nx), (ey[0], (ey[-1] - ey[0]) / ny, ny)
    for t, (m_ds, g_ds, _) in enumerate(pts):
        ref = O.binary_hess(m_ds, g_ds, E, Cm, y_index, (0, 1), imf, w.normalize_value,
                            O.imf_mean(imf), gx, gy)
        got = out[t].reshape(ny, nx).T
        assert ref.sum() > 0
        assert np.all(np.abs(got - ref) <= 1e-4 * np.abs(ref) + 1e-5 * np.abs(ref).max())
