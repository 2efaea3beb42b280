"""Timed cases of the library's public entry points.

Each case is a dict of plain values; prepare() makes its inputs from a seed, run() makes one
pass through the public API and returns the outputs whole, work() counts the bytes and
floating-point operations a pass cannot do without, and exact() gives the same outputs from
plain torch / numpy in 64 bits.

Paths ("path" of a case):
  templates   partial_cmd_smooth_batch: Hess-diagram templates of a grid of isochrones
  ragged_templates  partial_cmd_smooth_ragged: the same with one Hess grid per galaxy
  binary      binary_hess_batch: unresolved-binary templates
  fg          fg_: -logL, gradient and composite of one coefficient vector, host arrays
  fg_batched  fg_batched: many coefficient vectors on the tensor cores
  fg_ragged   fg_ragged: many galaxies with their own grids in one call
  fit         fit_templates_fast: a whole BFGS fit on the device
  emulator    TemplateEmulator.predict: templates from the per-cell networks and bases
  bin_cmd     bin_cmd: hard-binned catalogue
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..",
                                "starformationhistories.jl_gb300"))
import sfhgpu  # noqa: E402

XLIM, YLIM = (-0.6, 2.4), (19.0, 30.0)     # colour and magnitude window of the Hess diagrams
LOGAGE, MH = (6.6, 10.1), (-2.5, 0.3)      # log10(age / yr) and [M/H] of the template grids
DMOD = 25.0                                # distance modulus
ERR = (math.e, 1.0 / 1.2, 28.0 - 1.2 * math.log(0.3), 0.01)  # exp_photerr(m, a, b, c, d)
COMPL = (1.0, 28.0, 0.3)                   # Martin2016_complete(m, A, m50, rho)
IMF_SEG = ((0.08, 0.5, 1.3), (0.5, 100.0, 2.3))  # Kroupa (2001)


def listed():
    return [
        # a quick look at a handful of templates on a coarse grid (latency and launches)
        {"name": "templates_small", "path": "templates", "nt": 6, "nx": 40, "ny": 50,
         "n_iso": 120, "y_index": 1},
        # the production template grid of a fit: 40 ages x 30 metallicities, V against B - V
        {"name": "templates_production", "path": "templates", "nt": 1200, "nx": 200, "ny": 300,
         "n_iso": 400, "y_index": 1},
        # a magnitude outside the colour (R against B - V: independent errors), ragged sizes
        {"name": "templates_separable", "path": "templates", "nt": 300, "nx": 151, "ny": 213,
         "n_iso": 333, "y_index": 2},
        # a survey: galaxies with grids and isochrones of their own
        {"name": "ragged_templates", "path": "ragged_templates", "ngal": 64, "nt": 12,
         "nmin": 50, "nmax": 300, "imin": 100, "imax": 2000},
        # unresolved binaries mixed into a fit's templates
        {"name": "binary_templates", "path": "binary", "nt": 60, "nx": 200, "ny": 300,
         "n_iso": 400},
        # the objective of a small fit in Float64, host arrays (the smallest call: latency)
        {"name": "fg_float64_small", "path": "fg", "storage": "f64", "nt": 50, "nx": 75,
         "ny": 100, "stars": 1e4},
        # the objective of the production fit, FP32 templates, host arrays
        {"name": "fg_production", "path": "fg", "storage": "f32", "nt": 1200, "nx": 200,
         "ny": 300, "stars": 1e6},
        # the objective for all chains of a sampler at once
        {"name": "fg_batched_1024", "path": "fg_batched", "B": 1024, "nt": 1200, "nx": 200,
         "ny": 300, "stars": 1e6},
        # the objective of a survey's galaxies in one call
        {"name": "fg_ragged_256", "path": "fg_ragged", "ngal": 256, "nt": 12, "nmin": 50,
         "nmax": 300},
        # a whole fit (BFGS in sqrt space, the setting recommended for SFH fits)
        {"name": "fit_fast", "path": "fit", "nt": 240, "nx": 100, "ny": 150, "stars": 1e5},
        # emulated templates for a whole age-metallicity grid
        {"name": "emulator_predict", "path": "emulator", "B": 1200, "nx": 200, "ny": 300,
         "na": 16, "nm": 4, "K": 64},
        # an observed catalogue binned into its Hess diagram, host arrays in and out
        {"name": "bin_cmd_catalogue", "path": "bin_cmd", "n": 2_000_000, "nx": 200, "ny": 300,
         "weighted": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["templates", "templates", "ragged_templates", "binary", "fg", "fg",
                       "fg_batched", "fg_ragged", "fit", "emulator", "bin_cmd"])
    nx, ny = rng.randint(40, 200), rng.randint(50, 300)
    c = {"path": path}
    if path == "templates":
        c.update(nt=_log(rng, 6, 1200), nx=nx, ny=ny, n_iso=rng.randint(100, 400),
                 y_index=rng.choice([0, 1, 1, 2]))
    elif path == "ragged_templates":
        c.update(ngal=_log(rng, 4, 64), nt=rng.randint(2, 12), nmin=50,
                 nmax=rng.randint(80, 300), imin=100, imax=rng.randint(200, 2000))
    elif path == "binary":
        c.update(nt=_log(rng, 4, 60), nx=nx, ny=ny, n_iso=rng.randint(100, 400))
    elif path == "fg":
        if rng.random() < 0.5:
            c.update(storage="f64", nt=rng.randint(20, 200), nx=rng.randint(40, 100),
                     ny=rng.randint(50, 150), stars=10.0 ** rng.uniform(4, 5))
        else:
            c.update(storage="f32", nt=_log(rng, 100, 1200), nx=rng.randint(60, 200),
                     ny=rng.randint(80, 300), stars=10.0 ** rng.uniform(4, 6))
    elif path == "fg_batched":
        c.update(B=_log(rng, 64, 1024), nt=_log(rng, 50, 1200), nx=nx, ny=ny,
                 stars=10.0 ** rng.uniform(4, 6))
    elif path == "fg_ragged":
        c.update(ngal=_log(rng, 8, 256), nt=rng.randint(2, 30), nmin=50,
                 nmax=rng.randint(80, 220))
    elif path == "fit":
        c.update(nt=_log(rng, 30, 240), nx=rng.randint(50, 100), ny=rng.randint(60, 150),
                 stars=10.0 ** rng.uniform(4, 5))
    elif path == "emulator":
        c.update(B=_log(rng, 50, 1200), nx=nx, ny=ny, na=rng.randint(2, 16),
                 nm=rng.randint(1, 4), K=rng.choice([32, 48, 64]))
    else:
        c.update(n=_log(rng, 10_000, 2_000_000), nx=nx, ny=ny, weighted=rng.random() < 0.5)
    return c


# ------------------------------------------------------------------------------- inputs

def _edges(nx, ny):
    return np.linspace(*XLIM, nx + 1), np.linspace(*YLIM, ny + 1)


def _isochrone(la, mh, n):
    """(m_ini (n), magnitudes (3, n)) of a smooth analytic isochrone in (B, V, R)."""
    m = np.logspace(-1.0, math.log10(1.5), n)
    x, t = np.log10(m), la - 6.6
    g = 0.5 * (1.0 + np.tanh((x - (math.log10(1.45) - 0.07 * t)) / 0.02))
    V = 4.8 - 7.5 * x + 0.3 * t - 6.0 * g
    BV = 0.65 - 1.1 * x + 0.2 * mh + 0.9 * g * (1.0 - 0.3 * t / 3.5)
    return m, np.stack([V + BV, V, V - 0.55 * BV])


def _resample(m, mags, dmag, y_index):
    """Masses and magnitudes after inserting points until consecutive ones are at most dmag
    apart in the (B - V, magnitude) plane."""
    d = np.hypot(np.diff(mags[0] - mags[1]), np.diff(mags[y_index]))
    cnt = np.where(d > dmag, np.ceil(d / dmag), 1).astype(np.int64)
    k = np.repeat(np.arange(cnt.size), cnt)
    j = np.arange(k.size) - np.repeat(np.cumsum(cnt) - cnt, cnt) + 1
    c = cnt[k]
    mass = np.where(c == 1, m[k + 1], m[k] + (m[k + 1] - m[k]) / c * j)
    f = (mass - m[k]) / (m[k + 1] - m[k])
    new = mags[:, k] * (1.0 - f) + mags[:, k + 1] * f
    return np.concatenate([m[:1], mass]), np.concatenate([mags[:, :1], new], axis=1)


def _template_inputs(c, seed):
    """Per template: (m_ini, mags, dmod, (xedges, yedges)), on the host."""
    rng = np.random.default_rng(seed)
    if c["path"] == "ragged_templates":
        out = []
        for nx, ny, u in _ragged_shapes(c):
            n, dm = c["imin"] + int(u * (c["imax"] - c["imin"])), float(rng.uniform(24.5, 26.5))
            e = _edges(nx, ny)
            out += [(*_isochrone(rng.uniform(*LOGAGE), rng.uniform(*MH), n), dm, e)
                    for _ in range(c["nt"])]
        return out
    e, dm = _edges(c["nx"], c["ny"]), DMOD + float(rng.uniform(-0.3, 0.3))
    iso = [_isochrone(la, mh, c["n_iso"]) for la, mh in
           zip(np.sort(rng.uniform(*LOGAGE, c["nt"])), rng.uniform(*MH, c["nt"]))]
    if c["path"] == "binary":  # every fourth resampled point, shifted to the distance
        dmag = min((XLIM[1] - XLIM[0]) / c["nx"], (YLIM[1] - YLIM[0]) / c["ny"])
        iso = [(a[::4].copy(), b[:, ::4] + dm) for a, b in
               (_resample(m, g, dmag, 1) for m, g in iso)]
    return [(m, g, dm, e) for m, g in iso]


def _hess_matrix(nt, nx, ny, seed):
    """(nt, nbins) float64 CUDA templates: stars of growing error and falling weight along a
    curve through the Hess diagram, a bright sequence and a broad faint end."""
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(int(seed))
    P = 64
    u = torch.rand((nt, P), generator=g, device=dev, dtype=torch.float64)
    age = torch.linspace(0, 1, nt, device=dev, dtype=torch.float64)[:, None]
    met = torch.rand((nt, 1), generator=g, device=dev, dtype=torch.float64)
    y = 19.5 + 2.0 * age + (10.0 - 2.0 * age) * u
    x = 0.3 + 0.3 * met + 0.5 * (u - 0.4 - 0.3 * age) ** 2 + 0.15 * age
    s = 0.01 + 0.15 * torch.exp((y - 28.0) / 1.2)
    w = torch.exp(1.2 * (y - 26.0) / 2.5) / (1.0 + torch.exp((y - 28.0) / 0.3))

    def part(c, lim, n, sc):
        e = torch.linspace(lim[0], lim[1], n + 1, device=dev, dtype=torch.float64)
        t = torch.special.erf((e[None, None, :] - c[:, :, None]) / (math.sqrt(2.0) * sc[:, :, None]))
        return t[:, :, 1:] - t[:, :, :-1]
    X, Y = part(x, XLIM, nx, 1.4 * s), part(y, YLIM, ny, s) * w[:, :, None]
    M = torch.bmm(Y.transpose(1, 2), X).reshape(nt, ny * nx)  # column-major (nx, ny)
    return M + 1e-9


def _observed(M, stars, seed):
    """Coefficients that give `stars` stars and a Poisson draw of their composite (CUDA)."""
    g = torch.Generator(device=M.device).manual_seed(int(seed) + 1)
    r = torch.exp(torch.randn(M.shape[0], generator=g, device=M.device, dtype=torch.float64))
    m = r @ M
    r = r * (stars / m.sum())
    return r, torch.poisson(m * (stars / m.sum()), generator=g)


def _ragged_shapes(c):
    """Grid sizes of the galaxies and a uniform number for their isochrone lengths: part of
    the case, so outputs of every seed have one layout."""
    rng = np.random.default_rng(20261203)
    nxy = rng.integers(c["nmin"], c["nmax"] + 1, (c["ngal"], 2))
    return [(int(a), int(b), float(u)) for (a, b), u in zip(nxy, rng.random(c["ngal"]))]


def _fg_inputs(c, seed):
    M = _hess_matrix(c["nt"], c["nx"], c["ny"], seed)
    if c.get("storage") != "f64":
        M = M.float()
    r, data = _observed(M.double(), c["stars"], seed)
    g = torch.Generator(device=M.device).manual_seed(int(seed) + 2)
    shape = (c["B"], c["nt"]) if c["path"] == "fg_batched" else (c["nt"],)
    R = r * torch.exp(0.2 * torch.randn(shape, generator=g, device=M.device, dtype=torch.float64))
    return M, R, data


def _ragged_inputs(c, seed):
    Ms, rs, ds = [], [], []
    for k, (nx, ny, _) in enumerate(_ragged_shapes(c)):
        M = _hess_matrix(c["nt"], nx, ny, seed * 1000 + k).float()
        r, d = _observed(M.double(), 1e4, seed * 1000 + k)
        Ms.append(M)
        rs.append(1.1 * r)
        ds.append(d)
    return Ms, rs, ds


def _emulator_inputs(c, seed):
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(int(seed))
    G, K, nb = c["na"] * c["nm"], c["K"], c["nx"] * c["ny"]
    basis = 0.002 * torch.randn((G, K, nb), generator=g, device=dev)
    offset = 0.05 * torch.rand((G, nb), generator=g, device=dev)
    parts = []
    for fin, fout in ((3, 256), (256, 256), (256, K)):
        a = math.sqrt(6.0 / (fin + fout))
        parts += [a * (2 * torch.rand((G, fout * fin), generator=g, device=dev) - 1),
                  0.05 * torch.randn((G, fout), generator=g, device=dev)]
    lo, hi = np.array([6.6, -2.5, 24.95]), np.array([10.1, 0.3, 25.05])
    theta = lo + (hi - lo) * np.random.default_rng(seed).random((c["B"], 3))
    return basis, offset, torch.cat(parts, 1).reshape(-1), np.stack([lo, hi], 1), theta


def _catalogue(c, seed):
    rng = np.random.default_rng(seed)
    y = np.round(30.2 - rng.exponential(1.6, c["n"]), 3)
    x = np.round(0.3 + 0.05 * (y - 24.0) + rng.normal(0.0, 0.25, c["n"]), 3)
    return x, y, rng.random(c["n"]) if c["weighted"] else None


def prepare(case, seed):
    c = dict(case)
    path = c["path"]
    dev = torch.device("cuda", 0)
    st = {"c": c}
    if path in ("templates", "ragged_templates", "binary"):
        inp = _template_inputs(c, seed)
        lens = np.array([a.size for a, _, _, _ in inp], dtype=np.int32)
        st["off"] = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.int64)
        st["len"] = lens
        st["m"] = torch.as_tensor(np.concatenate([a for a, _, _, _ in inp]), device=dev)
        st["mags"] = torch.as_tensor(np.concatenate([b for _, b, _, _ in inp], axis=1), device=dev)
        st["dmod"] = np.array([d for _, _, d, _ in inp])
        st["edges"] = [e for _, _, _, e in inp]
        st["err"] = [sfhgpu.err_model(*ERR)] * 3
        st["compl"] = [sfhgpu.compl_model(*COMPL)] * 3
        st["imf"] = sfhgpu.Kroupa2001(0.08, 100.0)
    elif path in ("fg", "fit", "fg_batched"):
        M, R, data = _fg_inputs(c, seed)
        if path == "fg" and c["storage"] == "f64":
            st["H"] = sfhgpu.Models(M.cpu().numpy().T, storage="f64")
        else:
            torch.cuda.synchronize()
            st["H"] = sfhgpu.Models.from_device(
                M.data_ptr(), M.shape[1], c["nt"],
                storage="bf16x2" if path == "fg_batched" else "f32")
            st["H"].ctx.synchronize()
        if path == "fg_batched":
            st["R"], st["data"] = R, data
        else:
            st["r"], st["data"] = R.cpu().numpy(), data.cpu().numpy()
            st["G"], st["comp"] = np.empty(c["nt"]), np.empty(data.numel())
    elif path == "fg_ragged":
        Ms, rs, ds = _ragged_inputs(c, seed)
        packed = torch.cat([M.reshape(-1) for M in Ms])
        torch.cuda.synchronize()
        st["gal"] = sfhgpu.Galaxies(packed, [M.shape[1] for M in Ms], [M.shape[0] for M in Ms])
        st["r"], st["data"] = torch.cat(rs), torch.cat(ds)
    elif path == "emulator":
        basis, offset, params, bounds, theta = _emulator_inputs(c, seed)
        em = sfhgpu.TemplateEmulator(c["nx"] * c["ny"], ncomp=c["K"], bounds=bounds,
                                     basis_cells=(c["na"], c["nm"], 1))
        em.basis, em.offset, em.params = basis, offset, params
        st["em"], st["theta"] = em, theta
    else:
        st["x"], st["y"], st["w"] = _catalogue(c, seed)
        st["edges"] = (sfhgpu.julia_range(*XLIM, c["nx"] + 1), sfhgpu.julia_range(*YLIM, c["ny"] + 1))
    torch.cuda.synchronize()
    return st


# ------------------------------------------------------------------------------- one pass

def run(st):
    c = st["c"]
    path = c["path"]
    if path == "templates":
        return sfhgpu.partial_cmd_smooth_batch(
            st["m"], st["mags"], st["off"], st["len"], c["y_index"], (0, 1), st["err"],
            st["compl"], st["imf"], st["dmod"], 1.0, st["edges"][0])
    if path == "ragged_templates":
        return sfhgpu.partial_cmd_smooth_ragged(
            st["m"], st["mags"], st["off"], st["len"], 1, (0, 1), st["err"], st["compl"],
            st["imf"], st["dmod"], 1.0, st["edges"])[0]
    if path == "binary":
        return sfhgpu.binary_hess_batch(
            st["m"], st["mags"], st["off"], st["len"], 1, (0, 1), st["err"], st["compl"],
            st["imf"], 1.0, st["edges"][0])
    if path == "fg":
        v = sfhgpu.fg_(True, st["G"], st["r"], st["H"], st["data"], st["comp"])
        return {"value": v, "G": st["G"], "composite": st["comp"]}
    if path == "fg_batched":
        negL, G = sfhgpu.fg_batched(st["H"], st["R"], st["data"])
        return {"value": negL, "G": G}
    if path == "fg_ragged":
        negL, G, comp = sfhgpu.fg_ragged(st["gal"], st["r"], st["data"])
        return {"value": negL, "G": G, "composite": comp}
    if path == "fit":
        x, res = sfhgpu.fit_templates_fast(st["H"], st["data"], g_abstol=1e-3)
        return {"coeffs": x, "value": np.float64(res.fun)}
    if path == "emulator":
        return st["em"].predict(st["theta"])
    return sfhgpu.bin_cmd(st["x"], st["y"], weights=st["w"], edges=st["edges"]).weights


# ------------------------------------------------------------------------------- work

def _stamp_updates(c):
    """Bins that a template's stamps add to, estimated from a few of its templates."""
    inp = _template_inputs(dict(c, ngal=min(c.get("ngal", 0), 8), nt=min(c["nt"], 8)), 0)
    n = 0.0
    for m, g, dm, e in inp:
        x, y, sx, sy, _, cov = _stars(m, g, dm, e, c.get("y_index", 1))
        win = _window(x, y, sx, sy, cov, e)
        n += float(np.sum(np.where(win[4], (win[1] - win[0] + 1) * (win[3] - win[2] + 1), 0)))
    return n / len(inp)


def work(case):
    c = dict(case)
    path = c["path"]
    if path in ("templates", "binary", "ragged_templates"):
        inp = _template_inputs(c, 0)
        out = sum((e[0].size - 1) * (e[1].size - 1) for _, _, _, e in inp)
        pts = sum(a.size for a, _, _, _ in inp)
        if path == "binary":  # every pair of points: a weight and two magnitudes
            return {"bytes": 32.0 * pts + 4.0 * out,
                    "flops": sum(10.0 * a.size * a.size / 2 for a, _, _, _ in inp) + 2.0 * out}
        return {"bytes": 32.0 * pts + 4.0 * out, "flops": 2.0 * len(inp) * _stamp_updates(c)}
    nb = c.get("nx", 0) * c.get("ny", 0)
    if path == "fg":
        el = 8 if c["storage"] == "f64" else 4
        return {"bytes": el * nb * c["nt"] + 16.0 * nb + 16.0 * c["nt"],
                "flops": 4.0 * nb * c["nt"]}
    if path == "fg_batched":
        return {"bytes": 4.0 * nb * c["nt"] + 8.0 * nb + c["B"] * (12.0 * c["nt"] + 8.0),
                "flops": 4.0 * nb * c["nt"] * c["B"]}
    if path == "fg_ragged":
        nb = sum(a * b for a, b, _ in _ragged_shapes(c))
        return {"bytes": nb * (4.0 * c["nt"] + 16.0) + c["ngal"] * (16.0 * c["nt"] + 8.0),
                "flops": 4.0 * nb * c["nt"]}
    if path == "fit":  # at least one evaluation per template, a rank-two update after each
        return {"bytes": c["nt"] * (4.0 * nb * c["nt"] + 24.0 * c["nt"] ** 2),
                "flops": c["nt"] * (4.0 * nb * c["nt"] + 8.0 * c["nt"] ** 2)}
    if path == "emulator":
        cells = min(c["na"] * c["nm"], c["B"])
        return {"bytes": 4.0 * (cells * ((c["K"] + 1) * nb + 67000 + 257 * c["K"]) + c["B"] * nb),
                "flops": 2.0 * c["B"] * (c["K"] * nb + 66304 + 256 * c["K"])}
    return {"bytes": (24.0 if c["weighted"] else 16.0) * c["n"] + 8.0 * nb, "flops": 4.0 * c["n"]}


# ------------------------------------------------------------------------------- 64 bits

def _imf(m):
    """Kroupa (2001) density normalised on [0.08, 100] and its mean mass."""
    s, seg = 1.0, []
    for k, (lo, hi, a) in enumerate(IMF_SEG):
        if k:
            s *= lo ** (a - IMF_SEG[k - 1][2])
        seg.append((lo, hi, a, s))

    def integral(p):
        return sum(s_ * (hi ** (1 + p - a) - lo ** (1 + p - a)) / (1 + p - a)
                   for lo, hi, a, s_ in seg)
    pdf = np.where(m < 0.5, seg[0][3] * m ** -1.3, seg[1][3] * m ** -2.3) / integral(0)
    return pdf, integral(1) / integral(0)


def _err(m):
    return ERR[0] ** (ERR[1] * (m - ERR[2])) + ERR[3]


def _complete(m):
    return COMPL[0] / (1.0 + np.exp((m - COMPL[1]) / COMPL[2]))


def _stars(m, mags, dmod, e, y_index):
    """(x, y, sx, sy, weight, cov) of the stars a template's stamps are drawn for."""
    dmag = min((e[0][-1] - e[0][0]) / (e[0].size - 1), (e[1][-1] - e[1][0]) / (e[1].size - 1))
    mass, g = _resample(m, mags, dmag, y_index)
    g = g + dmod
    pdf, mean = _imf(mass)
    s = _err(g)
    comp = _complete(g[0]) * _complete(g[1])
    if y_index == 2:
        cov, cerr = 0, np.sqrt(s[0] ** 2 + s[1] ** 2)
        comp = comp * _complete(g[2])
    else:
        cov, cerr = (-1, s[1]) if y_index == 0 else (1, s[0])
    w = np.diff(mass) * (pdf[:-1] + pdf[1:]) / 2.0 * comp[:-1] / mean
    mid = [v[:-1] + np.diff(v) / 2.0 for v in (g[0] - g[1], g[y_index], cerr, s[y_index])]
    return (*mid, w, cov)


def _window(x, y, sx, sy, cov, e):
    """First and last bin (1-based) of each stamp on both axes, and whether it is drawn."""
    nx, ny = e[0].size - 1, e[1].size - 1
    xs, ys = (e[0][-1] - e[0][0]) / nx, (e[1][-1] - e[1][0]) / ny
    xc, yc = np.rint((x - e[0][0]) / xs + 1.0), np.rint((y - e[1][0]) / ys + 1.0)
    if cov == 0:
        xo = np.maximum(1, np.ceil(10.0 * sx / xs) // 2)
        yo = np.maximum(1, np.ceil(10.0 * sy / ys) // 2)
    else:
        xo = np.maximum(1, np.rint(15.0 * sx / xs / 2.0))
        yo = np.maximum(1, np.rint(10.0 * sy / ys / 2.0))
    x0, x1 = np.maximum(1, xc - xo), np.minimum(nx, xc + xo)
    y0, y1 = np.maximum(1, yc - yo), np.minimum(ny, yc + yo)
    return x0, x1, y0, y1, (x1 > x0) & (y1 > y0)


def _smooth(x, y, sx, sy, w, cov, e):
    """(ny * nx) float64 CUDA Hess diagram of weighted stars with Gaussian errors."""
    dev = torch.device("cuda", 0)
    nx, ny = e[0].size - 1, e[1].size - 1
    xs, ys = (e[0][-1] - e[0][0]) / nx, (e[1][-1] - e[1][0]) / ny
    x0, x1, y0, y1, ok = _window(x, y, sx, sy, cov, e)
    cols = [torch.as_tensor(np.ascontiguousarray(v[ok]), device=dev)
            for v in (x, y, sx, sy, w, x0, x1, y0, y1)]
    H = torch.zeros((ny, nx), dtype=torch.float64, device=dev)
    i = torch.arange(1, nx + 1, device=dev, dtype=torch.float64)
    j = torch.arange(1, ny + 1, device=dev, dtype=torch.float64)
    step = max(1, int(1.5e8 // (nx * ny)))
    r2 = math.sqrt(2.0)
    for a in range(0, cols[0].numel(), step):
        X, Y, SX, SY, W, A0, A1, B0, B1 = (v[a:a + step, None] for v in cols)
        inx, iny = (i >= A0) & (i <= A1), (j >= B0) & (j <= B1)
        if cov == 0:
            px, py = (X - e[0][0]) / xs + 1.0, (Y - e[1][0]) / ys + 1.0
            fx = torch.erf((i + 1 - px) / (r2 * SX / xs)) - torch.erf((i - px) / (r2 * SX / xs))
            fy = torch.erf((j + 1 - py) / (r2 * SY / ys)) - torch.erf((j - py) / (r2 * SY / ys))
            H += (0.25 * W * fy * iny).T @ (fx * inx)
            continue
        edge = (torch.arange(nx + 1, device=dev, dtype=torch.float64) * xs + e[0][0] - X)[:, None, :]
        for node, wt in ((-math.sqrt(0.6), 5.0 / 9.0), (0.0, 8.0 / 9.0), (math.sqrt(0.6), 5.0 / 9.0)):
            dy = (j - 0.5) * ys + e[1][0] - Y + node * ys / 2.0
            ck = W / (2.0 * math.sqrt(2.0 * math.pi) * SY) * (ys / 2.0) * wt * \
                torch.exp(-0.5 * (dy / SY) ** 2) * iny
            t = torch.erf((edge + cov * dy[:, :, None]) / (r2 * SX[:, :, None]))
            t = (t[:, :, 1:] - t[:, :, :-1]) * inx[:, None, :]
            H += torch.einsum("sj,sji->ji", ck, t)
    return H.reshape(-1)


def _pairs(m, g, e):
    """Weighted points of a template's unresolved binaries: pairs binned, one point per
    occupied bin."""
    nx, ny = e[0].size - 1, e[1].size - 1
    xs, ys = (e[0][-1] - e[0][0]) / nx, (e[1][-1] - e[1][0]) / ny
    pdf, mean = _imf(m)
    pre = 1.0 / mean / 4.0 / np.sum(np.diff(m) * (pdf[1:] + pdf[:-1]) / 2.0)
    i, j = np.triu_indices(m.size - 1, 1)
    flux = 10.0 ** (-0.4 * g[:2])
    b = -2.5 * np.log10(flux[:, i] + flux[:, j])
    q = np.diff(m) * (pdf[:-1] + pdf[1:])
    w = q[i] * q[j] * pre * _complete(b[0]) * _complete(b[1])
    kx = np.floor((b[0] - b[1] - e[0][0]) / xs).astype(np.int64)
    ky = np.floor((b[1] - e[1][0]) / ys).astype(np.int64)
    ok = (kx >= 0) & (kx < nx) & (ky >= 0) & (ky < ny)
    h = np.bincount(kx[ok] + nx * ky[ok], weights=w[ok], minlength=nx * ny)
    k = np.nonzero(h)[0]
    # bin centres are rounding ties of the stamp's pixel: the lower edge rounded once, plus
    # half a step, decides the pixel
    L = np.longdouble
    cx = ((k % nx) * L(xs) + L(e[0][0])).astype(np.float64) + xs / 2.0
    cy = ((k // nx) * L(ys) + L(e[1][0])).astype(np.float64) + ys / 2.0
    return cx, cy, _err(cy + cx), _err(cy), h[k], 1


def _fg64(M, r, data):
    """-logL, its gradient and 1 - n / c for templates M (nt, nbins), all float64."""
    c = torch.clamp(r @ M, min=2.220446049250313e-16)
    n = data
    t = torch.where(n > 0, n - c - n * torch.log(torch.where(n > 0, n, 1.0) / c), -c)
    w = 1.0 - n / c
    return -t.sum(-1), w @ M.T, w


def _bf(x):
    return x.to(torch.bfloat16).double()


def exact(case, seed):
    c = dict(case)
    path = c["path"]
    if path in ("templates", "ragged_templates"):
        if path == "templates" and c["y_index"] != 2 and c["nt"] * c["nx"] * c["ny"] > 5_000_000:
            return None  # minutes in 64 bits
        if path == "ragged_templates" and c["ngal"] * c["nt"] * c["nmax"] ** 2 > 10_000_000:
            return None
        out = []
        for m, g, dm, e in _template_inputs(c, seed):
            out.append(_smooth(*_stars(m, g, dm, e, c.get("y_index", 1)), e))
        return torch.cat(out) if path == "ragged_templates" else torch.stack(out)
    if path == "binary":
        return torch.stack([_smooth(*_pairs(m, g, e), e) for m, g, _, e in _template_inputs(c, seed)])
    if path == "fg":
        M, r, data = _fg_inputs(c, seed)
        v, G, w = _fg64(M.double(), r, data)
        return {"value": np.float64(v.item()), "G": G.cpu().numpy(), "composite": w.cpu().numpy()}
    if path == "fg_batched":
        M, R, data = _fg_inputs(c, seed)
        M = M.double()
        parts = [_fg64(M, R[k:k + 128], data) for k in range(0, c["B"], 128)]
        return {"value": torch.cat([p[0] for p in parts]), "G": torch.cat([p[1] for p in parts])}
    if path == "fg_ragged":
        got = [_fg64(M.double(), r, d) for M, r, d in zip(*_ragged_inputs(c, seed))]
        return {"value": torch.stack([v for v, _, _ in got]),
                "G": torch.cat([g for _, g, _ in got]), "composite": torch.cat([w for _, _, w in got])}
    if path == "fit":
        return None  # a minimiser's path, not a formula
    if path == "emulator":
        basis, offset, params, bounds, theta = _emulator_inputs(c, seed)
        G, K = c["na"] * c["nm"], c["K"]
        lo, hi = bounds[:, 0], bounds[:, 1]
        n = np.array([c["na"], c["nm"], 1])
        wd = (hi - lo) / n
        idx = np.clip(((theta - lo) / wd).astype(np.int64), 0, n - 1)
        x = torch.as_tensor((2.0 * (theta - (lo + idx * wd)) / wd - 1.0).astype(np.float32),
                            device=basis.device)
        grp = torch.as_tensor(idx[:, 0] * c["nm"] + idx[:, 1], device=basis.device)
        P = params.reshape(G, -1)[grp]
        a, at = x.double(), 0
        for fin, fout, last in ((3, 256, 0), (256, 256, 0), (256, K, 1)):
            Wt = _bf(P[:, at:at + fin * fout]).reshape(-1, fout, fin)
            at += fin * fout
            a = torch.bmm(Wt, _bf(a.float()).unsqueeze(2)).squeeze(2) + P[:, at:at + fout].double()
            at += fout
            a = a if last else 0.5 * a * (1.0 + torch.erf(a / math.sqrt(2.0)))
        out = torch.empty((c["B"], c["nx"] * c["ny"]), dtype=torch.float64, device=basis.device)
        for k in range(G):
            rows = torch.nonzero(grp == k).flatten()
            if rows.numel():
                out[rows] = torch.clamp(offset[k].double() + a[rows] @ basis[k].double(), min=0.0) ** 2
        return out
    x, y, w = _catalogue(c, seed)
    ex, ey = (np.array([(lo * 10 * (n - i) + hi * 10 * i) / (10 * n) for i in range(n + 1)])
              for (lo, hi), n in ((XLIM, c["nx"]), (YLIM, c["ny"])))
    kx, ky = (np.searchsorted(e, v, side="right") - 1 for e, v in ((ex, x), (ey, y)))
    ok = (kx >= 0) & (kx < c["nx"]) & (ky >= 0) & (ky < c["ny"])
    h = np.bincount(kx[ok] + c["nx"] * ky[ok], weights=None if w is None else w[ok],
                    minlength=c["nx"] * c["ny"])
    return h.astype(np.float64).reshape(c["ny"], c["nx"]).T
