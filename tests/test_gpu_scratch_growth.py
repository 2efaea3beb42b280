"""Template builds whose workspace grows between their two device passes: the first pass's results
are made anew, whatever address the larger block gets.

Tolerance, that of the template tests: per bin 1e-5 |ref| + 1e-6 max(ref)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batches():
    """Template batches of growing size, each larger than what the one before left reserved."""
    from sfhgpu import synthetic as S
    return [S.small(nages=a, nmh=b) for a, b in ((1, 1), (2, 2), (4, 6), (12, 12))]


def _build(sfh, w, ctx, ragged):
    import torch
    from sfhgpu import synthetic as S
    m_ini, mags, offs, lens = S.isochrone_batch(w)
    dev = torch.device("cuda", 0)
    args = (torch.tensor(m_ini, device=dev), torch.tensor(mags, device=dev), offs, lens, 1, (0, 1),
            S.error_models(), S.completeness_models(), S.imf(), w.dmod, w.normalize_value)
    if ragged:
        out = sfh.partial_cmd_smooth_ragged(*args, [(w.xedges, w.yedges)] * w.ntempl, ctx=ctx)[0]
    else:
        out = sfh.partial_cmd_smooth_batch(*args, (w.xedges, w.yedges), ctx=ctx)
    torch.cuda.synchronize()
    return out.cpu().numpy().reshape(w.ntempl, -1).astype(float)


@pytest.mark.parametrize("ragged", [False, True])
def test_builds_of_growing_size_on_one_context(sfh, O, ragged):
    from sfhgpu import synthetic as S
    ctx = sfh.Context(0)
    imf = O.kroupa2001()
    E = [O.ErrModel(e.a, e.b, e.c, e.d, e.cap) for e in S.error_models()]
    C = [O.ComplModel(c.A, c.m50, c.rho) for c in S.completeness_models()]
    for w in _batches():
        grown, again = _build(sfh, w, ctx, ragged), _build(sfh, w, ctx, ragged)
        peak = np.abs(again).max(axis=1, keepdims=True)
        assert np.all(peak > 0)
        assert np.all(np.abs(grown - again) <= 1e-5 * np.abs(again) + 1e-6 * peak)
        m, g, offs, lens = S.isochrone_batch(w)
        t = w.ntempl - 1
        sl = slice(offs[t], offs[t] + lens[t])
        nx, ny = w.grid
        ref = O.partial_cmd_smooth(m[sl], g[:, sl], E, C, 1, (0, 1), imf, w.dmod, w.normalize_value,
                                   O.imf_mean(imf), (w.xedges[0], (w.xedges[-1] - w.xedges[0]) / nx, nx),
                                   (w.yedges[0], (w.yedges[-1] - w.yedges[0]) / ny, ny))
        got = grown[t].reshape(ny, nx).T
        assert np.all(np.abs(got - ref) <= 1e-5 * np.abs(ref) + 1e-6 * np.abs(ref).max())
