"""fg! on FP64 templates against the FP64 oracle at the edges of the one-launch form: one bin to
past the matrix that fits one wave of 64-bin tiles, one template to several per thread.
Tolerance: FP64 sums of at most 2e4 terms, 1e-10 of the sum of their magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbins,nt", [(1, 1), (63, 3), (64, 64), (65, 127), (130, 128), (1000, 129),
                                      (7500, 50), (9728, 257), (19456, 20), (19457, 20), (9729, 399),
                                      (200, 256)])
def test_fg_float64(sfh, O, nbins, nt):
    rng = np.random.default_rng(nbins * 7 + nt)
    M = np.asfortranarray(rng.random((nbins, nt)) * rng.integers(0, 2, (nbins, 1)))
    r = np.exp(rng.standard_normal(nt))
    data = rng.poisson(M @ r).astype(float)
    H = sfh.Models(M, storage="f64")
    comp, G = np.empty(nbins), np.empty(nt)
    for _ in range(2):  # the counter of the last block is re-armed
        v = sfh.fg_(True, G, r, H, data, comp)
    v_ref, G_ref, c_ref = O.fg(r, M, data)
    c = np.maximum(M @ r, np.finfo(float).eps)
    w = 1 - data / c
    assert np.allclose(comp, w, rtol=1e-10, atol=1e-12)
    if np.isfinite(v_ref):
        terms = np.abs(data - c) + np.abs(data * np.log(np.where(data > 0, data, 1) / c))
        assert abs(v - v_ref) <= 1e-10 * max(terms.sum(), 1e-300)
    else:
        assert v == v_ref
    assert np.all(np.abs(G - G_ref) <= 1e-10 * (np.abs(M).T @ np.abs(w)) + 1e-300)
    # without -logL
    G2, comp2 = np.empty(nt), np.empty(nbins)
    assert sfh.fg_(None, G2, r, H, data, comp2) is None
    assert np.array_equal(G2, G) and np.array_equal(comp2, comp)
