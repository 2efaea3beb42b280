// templates.cu -- template (Hess diagram) construction on sm_103a.
//
// The stamp kernels replace bin_cmd_smooth (src/StarFormationHistories.jl:574-621) and
// the two addstar! methods (:345-408) with their kernels
// GaussianPSFAsymmetric / gaussian_int_general (:191-265) and
// GaussianPSFCovariant / gaussian_psf_covariant (:272-340).  A star takes one of three ways
// (star_record): where its kernel is so smooth that 8 x 8 Chebyshev points stand for 40 x 16
// bins (k_stamp_nodes); wide against the bins, 8 x 8 bins per lane in registers from 16
// exponentials and two FP32 operations per bin (k_stamp_tiles, wide_tile and mid_tile, which
// also interpolates the first and writes the template); the rest bin by bin, a warp per star,
// added in global memory (k_stamp_narrow).
// Window sizes, ties-to-even centroid rounding and the "both clipped lengths > 1" skip
// follow the reference exactly.  The bound is FP32 issue: 5.6e10 (star, bin) updates for
// 1,200 templates on 200 x 300 bins took 288 ms with nine exponentials and a shared-memory atomic
// per update, and 4.5 ms this way (tiles 2.4, nodes 0.8, star records 0.6, narrow stars 0.5); 300
// separable templates 8.3 -> 0.70 ms, 60 binary ones 10.3 -> 0.89 ms, 64 galaxies of 12 templates
// 180 -> 4.2 ms, 6 templates on 40 x 50 bins 475 -> 159 us.
//
// k_iso_stars replaces the single-star part of partial_cmd_smooth (:829-888):
// mini_spacing resampling (:110-148, block-wide prefix scan over segments),
// interpolate_mini (:77-81), exp_photerr / Martin2016 callables
// (src/utilities.jl:205,218), calculate_weights (:765-776), bias and midpoints
// (:417-436), emitting one star record per midpoint.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "sfh_internal.cuh"

namespace {

// Warps of a k_stamp_nodes CTA, which wait for one another at its end.  2, 4, 8, us: 1,200 templates
// 769, 759, 800; 768 of 64 galaxies 1,057, 854, 871; 60 binary ones 45, 28, 27.
constexpr int kNodeWarps = 4;
constexpr int kTileWarpsMax = 16;  // most warps of a k_stamp_tiles CTA
constexpr int kNarrowWarps = 4;   // warps of a k_stamp_narrow CTA
constexpr int kNarrowRows = 64;   // rows of a separable star's y table at a time

struct Grid2 {
    double xf, xs, yf, ys;
    int nx, ny;
    double ixs, iys;  // 1 / xs, 1 / ys
};

Grid2 make_grid(double xf, double xs, int64_t nx, double yf, double ys, int64_t ny) {
    return Grid2{xf, xs, yf, ys, (int)std::clamp<int64_t>(nx, 0, INT32_MAX),
                 (int)std::clamp<int64_t>(ny, 0, INT32_MAX), 1.0 / xs, 1.0 / ys};
}

// Signed erfc table entry: |value| = erfc(|t|), sign bit = sign of t.
__device__ __forceinline__ float erfc_signed(float t) { return copysignf(erfcf(fabsf(t)), t); }

// erf(tb) - erf(ta) from signed erfc entries, without cancellation when both edges sit in the
// same tail.
__device__ __forceinline__ float erf_diff(float ea, float eb) {
    const float a = fabsf(ea), b = fabsf(eb);
    if (signbit(ea) == signbit(eb)) return signbit(ea) ? b - a : a - b;
    const float d = (2.0f - a) - b;      // ta < 0 <= tb
    return signbit(ea) ? d : -d;         // tb < 0 <= ta: descending edges
}

// Gauss-Legendre 3-point weights, src/StarFormationHistories.jl:303-304.
__constant__ float c_glw[3] = {0.5555555555555556f, 0.8888888888888888f, 0.5555555555555556f};

// exp(-z^2) with the rounding error of z*z folded back in (z*z = p + e exactly).
__device__ __forceinline__ float exp_negsq(float z) {
    const float p = z * z;
    const float e = fmaf(z, z, -p);
    return expf(-p) * (1.0f - e);
}

// erf(ta + h) - erf(ta) = (2/√π) ∫ exp(-t²) dt over one bin, by 3-point Gauss-Legendre.
// Relative error < 3e-7 whenever h * max(1, |t|) <= 0.3 (checked against 50-digit erfc).
__device__ __forceinline__ float gl3_bin(float ta, float h) {
    const float hh = 0.5f * h, tm = ta + hh, d = 0.7745966692414834f * hh;
    return 1.1283791670955126f * hh *
           (0.5555555555555556f * (exp_negsq(tm - d) + exp_negsq(tm + d)) +
            0.8888888888888888f * exp_negsq(tm));
}

// Integral of the unit Gaussian kernel over one bin, erf(ta + h) - erf(ta): quadrature
// for bins narrow against the local scale (no cancellation), erfc differences otherwise.
__device__ __forceinline__ float gauss_bin(float ta, float h) {
    if (h * fmaxf(1.0f, fabsf(ta + 0.5f * h)) <= 0.3f) return gl3_bin(ta, h);
    return erf_diff(erfc_signed(ta), erfc_signed(ta + h));
}

__device__ __forceinline__ int64_t clamp_cut(double v) { return (int64_t)fmin(v, 4.0e9); }

// 2^x in one special-function instruction (relative error about 2^-22; results below the
// normal range become 0).
__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// ---------------------------------------------------------------- star records
// What the stamp loop needs of one star, in FP32: its clipped window and, by class, the
// numbers of its kernel.  The FP64 work (pixel rounding, window sizes, variances) is done
// once per star by one thread (k_iso_stars, k_bin_points, k_star_prep; by next_stars when the
// caller cannot size a record array): FP64 retires two operations per SM clock on this GPU.
enum { kStarNone = 0, kStarWide = 1, kStarMid = 2, kStarNarrow = 3 };

struct __align__(16) StarRec {
    // wide: hx, bx, by, amp | uref, vref, kx, ky | cu, cv, strips (64 bits)   (see wide_tile)
    // mid: hx, bx, by, amp | uref, vref, kx, du | dv, -, -, -      (see mid_tile)
    // narrow, covariant: uref, bx, bx low, sx | sx low, vref, by, pref | k4, uref low, vref low, by low
    // narrow, separable: invx, invy, dx0, dy0 | A/4
    float p[12];
    int xlo, xhi, ylo, yhi;  // first and last bin of the window, 0-based, inside the grid
    float ir, jr;            // reference bin (0-based; not of a separable narrow star)
    int cls, cov;
};

__device__ __forceinline__ unsigned long long star_strips(const StarRec &r) {
    return (unsigned long long)__float_as_uint(r.p[10]) |
           (unsigned long long)__float_as_uint(r.p[11]) << 32;
}
struct StarId {
    int32_t t, q;  // template, star of the template
};
// What decides whether a warp wants a wide or mid star: first and last row, strips (none of a mid
// star).  No rows for the other classes.
struct __align__(16) StarKey {
    int ylo, yhi;
    unsigned long long strips;
};
// bits lo .. hi
__device__ __forceinline__ unsigned long long strip_bits(int lo, int hi) {
    return (~0ull >> (63 - hi)) & (~0ull << lo);
}

// The Chebyshev tiles of a grid (smooth stars, see smooth_strips): wx x wy bins, in strips of
// wy rows, multiples of the 8 x 8 bin tile.  on: the grid has them.
struct Smooth {
    int on, wx, wy, nwc, nstrip;
    __host__ __device__ int tiles() const { return nwc * nstrip; }
    __host__ __device__ int groups() const { return (nwc * nstrip + 31) / 32; }
};

// At most 40 columns by 16 rows when the y step is 1.2 to 4 x steps, 40 rows below that, 8 above:
// about as far in units of sigma each way.  At most 64 strips (a star's mask).  Grids below
// 4,096 bins have none: the bin tiles of a template are then two warps' worth or less.
__host__ __device__ inline Smooth smooth_tiling(const Grid2 &g, bool want) {
    Smooth s{};
    const double q = fabs(g.ys / g.xs);
    s.wx = ((g.nx + (g.nx + 39) / 40 - 1) / ((g.nx + 39) / 40) + 7) / 8 * 8;
    s.nwc = (g.nx + s.wx - 1) / s.wx;
    s.wy = q <= 1.2 ? 40 : q <= 4.0 ? 16 : 8;
    const int least = ((g.ny + 63) / 64 + 7) / 8 * 8;
    if (s.wy < least) s.wy = least;
    s.nstrip = (g.ny + s.wy - 1) / s.wy;
    s.on = want && (int64_t)g.nx * g.ny >= 4096;
    return s;
}

constexpr float kRoot2G = 1.1774100225154747f;  // sqrt 2 / g: u in units of sigma

// The record of one star: GaussianPSFAsymmetric / GaussianPSFCovariant windows as in
// addstar! (:345-408), then the class.
//
// The integral of a Gaussian over a bin is the Gaussian with the box's variance (step^2 / 12)
// added to its own, times 1 - step^4 / (2880 sigma^4) He4 (the box's fourth cumulant), up to
// sixth order in step / sigma.  With the base-2 scale g = sqrt(log2 e) folded in, a bin's
// value is amp 2^-(u^2 + v^2) times the correction, u and v linear in the bin's indices.
//
// Wide stars (both steps small against the kernel): the box on both axes.  Covariant kernel:
// the line at 0.08 (y steps in quadrature) and 0.045 (x step), in units of sqrt 2 sigma, keeps
// the form, with its correction taken to second order over a tile, within 5e-8 of the kernel's
// peak and 9e-7 of a bin's own value down to 1e-4 of the peak, against the reference's
// 3-point rule in 64 bits.  Separable kernel: 0.1 on each axis (the correction is taken at
// every row and column; sixth-order terms stay below 1e-9 of the peak).
//
// Mid stars (covariant kernel, x step small only): the box in x, the reference's three
// Gauss-Legendre nodes in y as they are.  x step up to 0.1, and x step^2 * y shift up to
// 2.5e-3 so that one correction serves the three nodes (y step up to 4): within 1e-8 of the peak and 1.5e-6
// of a bin's own value down to 1e-4 of the peak.  The rest (a few bins per sigma) is integrated
// bin by bin with erfc differences.
//
// FP64 throughput bounds this: divisions and square roots in full were three quarters of it.
// Quantities that only need FP32 results take one Newton step from an FP32 seed (2^-44); pixel
// numbers and window sizes take the product with the grid's inverse step, and the exact
// division only within 1e-9 of a rounding boundary.
__device__ __forceinline__ double rsqrt_nr(double v) {
    if (!(v > 1.0e-30 && v < 1.0e30)) return 1.0 / sqrt(v);
    const double y = (double)rsqrtf((float)v);
    return fma(0.5 * y, fma(-(v * y), y, 1.0), y);
}
__device__ __forceinline__ double rcp_nr(double v) {
    const double a = fabs(v);
    if (!(a > 1.0e-30 && a < 1.0e30)) return 1.0 / v;
    const double y = (double)__frcp_rn((float)v);
    return fma(y, fma(-v, y, 1.0), y);
}
// z, or exact() when z is within 1e-9 of half way between integers (half) / of an integer.
template <bool HALF, typename F>
__device__ __forceinline__ double near_exact(double z, F exact) {
    const double d = fabs(z - rint(z)), tol = fma(1.0e-9, fabs(z), 1.0e-9);
    const bool safe = HALF ? d < 0.5 - tol : d > tol;
    return safe ? z : exact();
}

__device__ __forceinline__ void star_record(StarRec &r, const Grid2 &g, double x, double y,
                                            double sx, double sy, double A, int cov) {
    r.cls = kStarNone;
    r.cov = cov;
    r.xlo = r.ylo = 0;
    r.xhi = r.yhi = -1;
    if (!(sx >= 0.0 && sy >= 0.0)) return;
    // histogram_pix, :502
    const double x0 = near_exact<true>(fma(x - g.xf, g.ixs, 1.0), [&] { return (x - g.xf) / g.xs + 1.0; });
    const double y0 = near_exact<true>(fma(y - g.yf, g.iys, 1.0), [&] { return (y - g.yf) / g.ys + 1.0; });
    if (!(fabs(x0) < 4.0e15 && fabs(y0) < 4.0e15)) return;
    const int64_t xc = __double2ll_rn(x0), yc = __double2ll_rn(y0);  // round(Int, ·): ties to even
    const double ssx = sx * g.ixs, ssy = sy * g.iys;
    int64_t xoff, yoff;
    if (cov == 0) {
        // size(GaussianPSFAsymmetric) = (ceil(Int, 10σx), ceil(Int, 10σy)), :247
        if (!(ssx >= 0.0 && ssy >= 0.0)) return;
        const double cx = near_exact<false>(10.0 * ssx, [&] { return sx / g.xs * 10.0; });
        const double cy = near_exact<false>(10.0 * ssy, [&] { return sy / g.ys * 10.0; });
        xoff = max((int64_t)1, clamp_cut(ceil(cx)) / 2);
        yoff = max((int64_t)1, clamp_cut(ceil(cy)) / 2);
    } else {
        // size(GaussianPSFCovariant) = (15σx, 10σy), :293; half widths, :383-384
        const double cx = near_exact<true>(7.5 * ssx, [&] { return 15.0 * sx / g.xs / 2.0; });
        const double cy = near_exact<true>(5.0 * ssy, [&] { return 10.0 * sy / g.ys / 2.0; });
        xoff = max((int64_t)1, (int64_t)__double2ll_rn(fmin(cx, 4.0e9)));
        yoff = max((int64_t)1, (int64_t)__double2ll_rn(fmin(cy, 4.0e9)));
    }
    const int64_t xlo = max((int64_t)1, xc - xoff), xhi = min((int64_t)g.nx, xc + xoff);
    const int64_t ylo = max((int64_t)1, yc - yoff), yhi = min((int64_t)g.ny, yc + yoff);
    if (!(xhi - xlo + 1 > 1 && yhi - ylo + 1 > 1)) return;  // :359, :401
    r.xlo = (int)xlo - 1;
    r.xhi = (int)xhi - 1;
    r.ylo = (int)ylo - 1;
    r.yhi = (int)yhi - 1;
    r.cls = kStarNarrow;
    const float xsf = (float)g.xs, ysf = (float)g.ys;
    const float hx = 0.70710678f * xsf / (float)sx, by = 0.70710678f * ysf / (float)sy;
    const float bx = cov ? 0.70710678f * ysf / (float)sx : 0.f;
    // (a weight that is not a finite float stays bin by bin: 0 * inf must not leave the window)
    const bool fine = fabs(A) <= 1.0e30 && hx > 0.f && by > 0.f;
    const bool wide = fine && (cov ? hx <= 0.045f && bx * bx + by * by <= 0.08f * 0.08f
                                   : hx <= 0.1f && by <= 0.1f);
    const bool mid = fine && cov != 0 && !wide && hx <= 0.1f && hx * hx * bx <= 2.5e-3f && by <= 4.f;
    const double c = (double)cov, gs = 1.2011224087864498;  // sqrt(log2 e)
    // the star's offset from its reference bin: its own, moved into its window
    const int irl = (int)min(max(xc, xlo), xhi), jrl = (int)min(max(yc, ylo), yhi);
    const double X = fma((double)irl - 0.5, g.xs, g.xf - x), Y = fma((double)jrl - 0.5, g.ys, g.yf - y);
    r.ir = (float)(irl - 1);
    r.jr = (float)(jrl - 1);
    if (wide || mid) {
        const double sy2 = sy * sy, Syy = wide ? fma(g.ys * (1.0 / 12.0), g.ys, sy2) : sy2;
        const double ry = rsqrt_nr(Syy), s2 = sy2 * (ry * ry), m = wide ? -c * s2 : -c;
        // the y box's share c^2 sy^2 - (c sy^2)^2 / Syy as a product: the difference loses vx where sy >> sx
        const double box = wide ? c * c * s2 * (g.ys * g.ys * (1.0 / 12.0)) : 0.0;
        const double vx = fma(sx, sx, fma(g.xs * (1.0 / 12.0), g.xs, box));
        const double rx = rsqrt_nr(vx), qx = 0.8493218002880191 * rx, qy = 0.8493218002880191 * ry;  // g / √2
        const double wsh = -m * g.ys * qx;
        const float wxf = (float)(g.xs * qx), wshf = (float)wsh, wyf = (float)(g.ys * qy);
        const float uref = (float)((X - m * Y) * qx), vref = (float)(Y * qy);
        // 2^(exponents relative to a tile's centre) stays in range over the window
        const float eu = (float)(xhi - xlo + 1) * wxf + (float)(yhi - ylo + 1) * fabsf(wshf) + fabsf(uref);
        const float ev = (float)(yhi - ylo) * wyf + fabsf(vref);
        if (eu * wxf <= 10.f && (mid ? fabsf(wshf) * wxf <= 1.f : eu * fabsf(wshf) + ev * wyf <= 10.f)) {
            const float rxf = (float)rx, k4x = xsf * rxf * (xsf * rxf);
            const double amp = A * (g.xs * rx) * (g.ys * ry) * 0.15915494309189535;  // A dx dy / (2π √(vx Syy))
            r.cls = wide ? kStarWide : kStarMid;
            r.p[0] = wxf;
            r.p[1] = wshf;
            r.p[2] = wyf;
            r.p[4] = uref;
            r.p[5] = vref;
            r.p[6] = k4x * k4x * (1.f / 2880.f);
            if (wide) {
                const float ryf = (float)ry, mf = (float)m, P = fmaf(mf * rxf, mf * rxf, ryf * ryf);
                const float s = rsqrtf(P), k4y = ysf * ysf * P;
                r.p[3] = (float)amp;
                r.p[7] = k4y * k4y * (1.f / 2880.f);
                r.p[8] = -1.1774100225f * s * mf * rxf;  // sqrt 2 / g
                r.p[9] = 1.1774100225f * s * ryf;
                r.p[10] = r.p[11] = 0.f;  // no smooth strips
            } else {
                r.p[3] = (float)(amp * 0.4444444444444444);  // weight 8/9 of the middle node, halved
                r.p[7] = (float)(0.3872983346207417 * wsh);  // sqrt(3/5) / 2 row
                r.p[8] = (float)(0.3872983346207417 * (g.ys * qy));
            }
            return;
        }
    }
    if (cov == 0) {
        // Bin i spans pixel coordinates [i, i+1]: evaluate at i + 1/2 with half width 1/2.
        r.p[0] = (float)(0.7071067811865476 * g.xs * rcp_nr(sx));
        r.p[1] = (float)(0.7071067811865476 * g.ys * rcp_nr(sy));
        r.p[2] = (float)((double)xlo - x0);
        r.p[3] = (float)((double)ylo - y0);
        r.p[4] = (float)(A * 0.25);
        return;
    }
    // A few bins per sigma (x step up to 0.25 sqrt 2 sigma): a bin's x integral as the Gaussian
    // with the box's variance, corrected through its sixth cumulant (He8 terms below 3e-9);
    // u at bin centres, base-2 scale.  Else erfc differences, u = t at the bins' lower edges.
    const bool gauss = hx > 0.f && hx <= 0.25f;
    const double rx = rsqrt_nr(gauss ? fma(sx, sx, g.xs * g.xs * (1.0 / 12.0)) : sx * sx);
    // (a vanishing error: far edges at a large finite t, a hard histogram)
    const double scale = fmin(0.7071067811865476 * rx * (gauss ? gs : 1.0), 1.0e30);
    const double bxs = c * g.ys * scale, sxs = g.xs * scale;
    const double uref = (X + c * Y - (gauss ? 0.0 : g.xs * 0.5)) * scale;
    r.p[0] = (float)uref;
    r.p[9] = (float)(uref - (double)r.p[0]);
    r.p[1] = (float)bxs;
    r.p[2] = (float)(bxs - (double)r.p[1]);
    r.p[3] = (float)sxs;
    r.p[4] = (float)(sxs - (double)r.p[3]);
    const double isy = rcp_nr(sy) * 0.8493218002880191, vref = Y * isy, bys = g.ys * isy;
    r.p[5] = (float)vref;
    r.p[6] = (float)bys;
    r.p[10] = (float)(vref - (double)r.p[5]);
    r.p[11] = (float)(bys - (double)r.p[6]);
    // prefac = A / 2 / sqrt(2π) / σy (:320) times the scale hy = dy / 2 of the GL weights
    // (:325), and the unit Gaussian's integral 2/√π dx / (√2 √vx)
    const double k = g.xs * rx;
    r.p[7] = (float)(A * bys * 0.11742965983745643 * (gauss ? 0.7978845608028654 * k : 1.0));
    const float k2 = (float)(k * k);
    r.p[8] = gauss ? k2 * k2 * (1.f / 2880.f) : -1.f;
}

// The strips over which a wide star's contribution can be interpolated from 8 x 8 Chebyshev
// points per tile: its window covers the strip, and over a tile's half width its logarithm
// changes by at most 0.7 on each axis, 0.08 of it by curvature.  The interpolation error of
// exp(c x) is 2 (c/2)^8 / 8! = 1e-8 of the value at the tile's centre, that of exp(-q x^2)
// 2 (q/4)^4 / 4! = 1.3e-8; at the tile's far end it is e^0.8 times that of the value there.
__device__ __forceinline__ unsigned long long smooth_strips(const StarRec &r, const Grid2 &g,
                                                            const Smooth &sm) {
    if (r.xlo > 0 || r.xhi < g.nx - 1) return 0ull;
    const float xh = 0.5f * (float)sm.wx, yh = 0.5f * (float)sm.wy;
    const float hx = r.p[0], bx = r.p[1], by = r.p[2], ln2 = 0.6931472f;
    if (!(ln2 * hx * hx * xh * xh <= 0.08f && ln2 * (bx * bx + by * by) * yh * yh <= 0.08f)) return 0ull;
    unsigned long long m = 0ull;
    const float i0 = -r.ir - 0.5f, i1 = i0 + (float)(sm.nwc * sm.wx);
    const float u0 = fmaf(i0, hx, r.p[4]), u1 = fmaf(i1, hx, r.p[4]);
    for (int k = 0; k < sm.nstrip; ++k) {
        const int ra = k * sm.wy, rb = min(g.ny, ra + sm.wy) - 1;
        if (r.ylo > ra || r.yhi < rb) continue;
        // u and v are linear: largest magnitudes at the corners of the area the tiles cover
        const float j0 = (float)ra - r.jr - 0.5f, j1 = j0 + (float)sm.wy;
        const float um = fmaxf(fmaxf(fabsf(fmaf(j0, bx, u0)), fabsf(fmaf(j1, bx, u0))),
                               fmaxf(fabsf(fmaf(j0, bx, u1)), fabsf(fmaf(j1, bx, u1))));
        const float vm = fmaxf(fabsf(fmaf(j0, by, r.p[5])), fabsf(fmaf(j1, by, r.p[5])));
        if (2.f * ln2 * um * hx * xh <= 0.7f && 2.f * ln2 * (um * fabsf(bx) + vm * by) * yh <= 0.7f)
            m |= 1ull << k;
    }
    return m;
}

// Completes a star's record with its smooth strips, stores it and its key, and lists it when it is narrow:
// the narrow stars of all templates are in one list (one atomic per warp).
__device__ __forceinline__ void store_record(StarRec &r, const Grid2 &g, StarId id, StarRec *to, StarKey *key,
                                             StarId *narrow, int *n_narrow, bool smooth = true) {
    unsigned long long m = 0ull;
    if (r.cls == kStarWide) {
        const Smooth sm = smooth_tiling(g, smooth);
        m = sm.on ? smooth_strips(r, g, sm) : 0ull;
        r.p[10] = __uint_as_float((unsigned int)m);
        r.p[11] = __uint_as_float((unsigned int)(m >> 32));
    }
    const unsigned act = __activemask(), nar = __ballot_sync(act, r.cls == kStarNarrow);
    if (r.cls == kStarNarrow) {
        const int lane = threadIdx.x & 31, lead = __ffs(nar) - 1;
        int at = 0;
        if (lane == lead) at = atomicAdd(n_narrow, __popc(nar));
        at = __shfl_sync(nar, at, lead);
        narrow[at + __popc(nar & ((1u << lane) - 1u))] = id;
    }
    *to = r;
    *key = r.cls == kStarWide || r.cls == kStarMid ? StarKey{r.ylo, r.yhi, m} : StarKey{INT_MAX, -1, 0ull};
}

constexpr int kPrepThreads = 64;  // small blocks: a few hundred stars already spread over the SMs

__global__ void __launch_bounds__(kPrepThreads)
k_star_prep(const double *__restrict__ xs, const double *__restrict__ ys,
            const double *__restrict__ sxs, const double *__restrict__ sys,
            const double *__restrict__ ws, const int64_t *__restrict__ start,
            const int32_t *__restrict__ count, const int32_t *__restrict__ covs, Grid2 g0,
            const Grid2 *__restrict__ grids, int t0, bool smooth, StarRec *__restrict__ rec,
            StarKey *__restrict__ key, StarId *__restrict__ narrow, int *__restrict__ n_narrow) {
    const int t = t0 + blockIdx.y;
    const int q = blockIdx.x * kPrepThreads + threadIdx.x;
    if (q >= count[t]) return;
    const int64_t s = start[t] + q;
    StarRec r{};
    const Grid2 g = grids ? grids[t] : g0;
    star_record(r, g, xs[s], ys[s], sxs[s], sys[s], ws[s], covs[t]);
    store_record(r, g, StarId{t, q}, rec + s, key + s, narrow, n_narrow, smooth);
}

// ---------------------------------------------------------------- narrow stars
// A star whose kernel is not wide against the bins: a warp adds it to the template in global
// memory (L2 adds FP32 natively; a shared-memory FP32 atomicAdd is a compare-and-swap loop).
// Separable kernel: x and y factor tables.
__device__ void star_asym(float *__restrict__ out, float *bx_buf, float *by_buf, const StarRec &r,
                          int nx, int lane) {
    const int lx = r.xhi - r.xlo + 1;
    const float invx = r.p[0], invy = r.p[1], dx0 = r.p[2], dy0 = r.p[3], a4 = r.p[4];
    // segments of W columns, each lane on its column: a product and an add per bin (a bin's row and
    // column from its number took two conversions, 16 a clock: 262 us for the narrow stars of
    // 300 separable templates on 151 x 213 bins, 230 us this way in the same grid of blocks)
    const int W = (lx + (lx + 31) / 32 - 1) / ((lx + 31) / 32), rows_per = 32 / W;
    const int seg = lane / W, pos = lane - seg * W;
    for (int m = lane; m < lx; m += 32) bx_buf[m] = gauss_bin((dx0 + (float)m) * invx, invx);
    for (int j0 = r.ylo; j0 <= r.yhi; j0 += kNarrowRows) {
        const int ly = min(kNarrowRows, r.yhi - j0 + 1);
        for (int m = lane; m < ly; m += 32)
            by_buf[m] = a4 * gauss_bin((dy0 + (float)(m + j0 - r.ylo)) * invy, invy);
        __syncwarp();
        if (seg < rows_per)
            for (int e = pos; e < lx; e += W) {
                const float x = bx_buf[e];
                float *to = out + (int64_t)(j0 + seg) * nx + r.xlo + e;
#pragma unroll 4
                for (int j = seg; j < ly; j += rows_per, to += (int64_t)rows_per * nx)
                    atomicAdd(to, x * by_buf[j]);
            }
        __syncwarp();
    }
}

// Covariant kernel.  Each lane prepares one row: per Gauss-Legendre node in y its weight, and
// u of a bin near the kernel's centre in that row (the shear and the bin's offset cancel there:
// their sum is formed in two floats), which the warp then reads by shuffles.
__device__ void star_cov(float *__restrict__ out, const StarRec &r, int nx, int lane) {
    const float sx = r.p[3], k4 = r.p[8], k6 = 0.85183542f * fmaxf(k4, 0.f) * sqrtf(fmaxf(k4, 0.f));  // k^4 / 2880, k^6 / 181440
    const int lx = r.xhi - r.xlo + 1, nrows = r.yhi - r.ylo + 1;
    const float c_first = (float)r.xlo - r.ir, c_last = (float)(r.xhi + 1) - r.ir;
    float *row0 = out + (int64_t)r.ylo * nx + r.xlo;
    const bool gauss = k4 >= 0.f;
    // 1 - k4 He4(z) + k6 He6(z), z^2 = 2 ln 2 u^2, by powers of u^2
    const float g0 = 1.f - 3.f * k4 - 15.f * k6, g1 = 1.3862943611198906f * (6.f * k4 + 45.f * k6);
    const float g2 = -1.9218120556728056f * (k4 + 15.f * k6), g3 = 2.6641971970211f * k6;
    const int W = min(gauss ? lx : lx + 1, 32), rows_per = 32 / W;
    const int nb = gauss ? W : W - 1;  // bins per segment pass
    const int seg = lane / W, pos = lane - seg * W;
    for (int r0 = 0; r0 < nrows; r0 += 32) {
        float ck[3], tk[3], ek[3];
        // u (at the reference bin) and v of the row's centre as two floats each
        const float d = (float)(r.ylo + r0 + lane) - r.jr, bx = r.p[1], by = r.p[6];
        const float p = d * bx, uh = r.p[0] + p, z = uh - r.p[0];
        const float ul = ((r.p[0] - (uh - z)) + (p - z)) + fmaf(d, r.p[2], fmaf(d, bx, -p) + r.p[9]);
        const float p2 = d * by, vh = r.p[5] + p2, z2 = vh - r.p[5];
        const float vl = ((r.p[5] - (vh - z2)) + (p2 - z2)) +
                         fmaf(d, r.p[11], fmaf(d, by, -p2) + r.p[10]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float gk = (float)(k - 1) * 0.38729835f, gl = (float)(k - 1) * -1.0945054e-8f;  // sqrt(3/5) / 2
            // uh + gk bx as two floats: a y step of thousands of x sigmas leaves no bits to either
            const float g = gk * bx, s = uh + g, zs = s - uh;
            const float sl = ((uh - (s - zs)) + (g - zs)) + fmaf(gk, r.p[2], fmaf(gk, bx, -g));
            ek[k] = fminf(fmaxf(rintf(-__fdividef(s, sx)), c_first), c_last);
            tk[k] = fmaf(ek[k], sx, s) + (sl + fmaf(gl, bx, fmaf(ek[k], r.p[4], ul)));
            const float v = fmaf(gk, by, vh) + fmaf(gl, by, fmaf(gk, r.p[11], vl)), q = v * v;
            ck[k] = r.p[7] * c_glw[k] * ex2f(-q) * fmaf(-0.6931471805599453f, fmaf(v, v, -q), 1.f);
        }
        const int rend = min(32, nrows - r0);
        for (int rb = 0; rb < rend; rb += rows_per) {
            const int row = rb + seg;
            const bool vrow = seg < rows_per && row < rend;
            float c[3], t0[3], e0k[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                c[k] = __shfl_sync(0xffffffffu, ck[k], row & 31);
                t0[k] = __shfl_sync(0xffffffffu, tk[k], row & 31);
                e0k[k] = __shfl_sync(0xffffffffu, ek[k], row & 31) - c_first;
            }
            for (int e0 = 0; e0 < lx; e0 += nb) {
                const int e = e0 + pos;
                float v = 0.f;
                bool put = vrow && e < lx;
                if (gauss) {
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const float u = fmaf((float)e - e0k[k], sx, t0[k]), q = u * u;
                        v = fmaf(c[k] * ex2f(-q), fmaf(q, fmaf(q, fmaf(q, g3, g2), g1), g0), v);
                    }
                } else {
                    float ev[3];
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        ev[k] = vrow && e <= lx ? erfc_signed(fmaf((float)e - e0k[k], sx, t0[k])) : 0.f;
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const float en = __shfl_down_sync(0xffffffffu, ev[k], 1);
                        v = fmaf(c[k], erf_diff(ev[k], en), v);
                    }
                    put = put && pos < W - 1;
                }
                if (put) atomicAdd(row0 + (int64_t)(r0 + row) * nx + e, v);
            }
        }
    }
}

// ---------------------------------------------------------------- wide stars
// One lane's 8 x 8 tile of bins in registers (acc[row][column pair]).  About the tile's
// centre (u, v),
//   u^2 + v^2 at (di, dj) = (u^2 + v^2) + 2 u hx di + hx^2 di^2
//                           + 2 (u bx + v by) dj + (bx^2 + by^2) dj^2 + 2 hx bx di dj,
// so the bin's value is X[di] Y[dj] T[dj][di]: 8 + 8 exponentials per tile, T (the star's
// own shear table, shared by all tiles) from shared memory, and a multiply and an FMA per
// bin on packed pairs (no T for the separable kernel).  The He4 corrections of the covariant
// kernel enter X and Y by their value, slope and axial curvature at the tile's centre, those
// of the separable kernel at every row and column.  X and Y are zero
// outside the star's window.
//
// NODES: the same at the 8 x 8 Chebyshev points of a larger tile that the star's window
// covers (see smooth_strips): the values are interpolated to the bins once, after the sum
// over stars.  Each (star, strip) is taken by one of the two forms.
__device__ __forceinline__ float tile_node(bool nodes, int i) {  // ascending, i = 0..7
    if (!nodes) return (float)i - 3.5f;
    const int k = i < 4 ? i : 7 - i;
    const float c = k == 0 ? 0.9807852804032304f : k == 1 ? 0.8314696123025452f
                  : k == 2 ? 0.5555702330196022f : 0.19509032201612825f;
    return i < 4 ? -c : c;
}

// The bits of 0 .. 7 from lo to hi (any two ints, lo <= hi).
__device__ __forceinline__ unsigned window_bits(int lo, int hi) {
    return (0xffu << min(max(lo, 0), 8)) & (0xffu >> (7 - min(max(hi, -1), 7))) & 0xffu;
}

struct Tile {
    int col0, row0;          // first bin (plain tiles)
    float xc, yc, xh, yh;    // centre in 0-based bins, half widths (NODES)
    int strip;               // the strip it lies in
    bool live;
};

template <bool COV, bool NODES>
__device__ __forceinline__ void wide_tile(float2 (&acc)[8][4], const StarRec &r,
                                          const float *__restrict__ T, const Tile &tl) {
    const int col0 = tl.col0, row0 = tl.row0;
    const bool own = ((star_strips(r) >> tl.strip & 1ull) != 0ull) == NODES;
    const bool over = tl.live && own && (NODES || (col0 <= r.xhi && col0 + 7 >= r.xlo &&
                                                   row0 <= r.yhi && row0 + 7 >= r.ylo));
    if (!__any_sync(0xffffffffu, over)) return;
    const bool part = !NODES && over && !(col0 >= r.xlo && col0 + 7 <= r.xhi && row0 >= r.ylo &&
                                          row0 + 7 <= r.yhi);
    // a lane outside the window works on the reference bin with amplitude 0
    const float di0 = over ? (NODES ? tl.xc : (float)col0 + 3.5f) - r.ir : 0.f;
    const float dj0 = over ? (NODES ? tl.yc : (float)row0 + 3.5f) - r.jr : 0.f;
    const float amp = over ? r.p[3] : 0.f;
    float u = fmaf(di0, r.p[0], r.p[4]);
    if (COV) u = fmaf(dj0, r.p[1], u);
    const float v = fmaf(dj0, r.p[2], r.p[5]);
    const float hx = NODES ? r.p[0] * tl.xh : r.p[0], bx = NODES ? r.p[1] * tl.yh : r.p[1];
    const float by = NODES ? r.p[2] * tl.yh : r.p[2];
    // u^2 + v^2 with its rounding error e
    const float pu = u * u, pv = v * v, s = pu + pv, z = s - pu;
    const float e = (fmaf(u, u, -pu) + fmaf(v, v, -pv)) + ((pu - (s - z)) + (pv - z));
    const float zx = kRoot2G * u;
    float X[8], A, gy, cy, zy = 0.f;  // row j: A 2^(gy d - cy d^2)
    if (COV || NODES) {
        // 1 - kx He4(zx) - ky He4(xi) at the centre: its value, and of its logarithm (base 2)
        // the slopes (4 log2 e He3) and the curvature along the two axes (6 log2 e He2)
        const float kx = r.p[6], ky = r.p[7], cu = r.p[8], cv = r.p[9];
        const float xi = fmaf(cu, u, cv * v), zx2 = zx * zx, xi2 = xi * xi;
        const float lr = -fmaf(kx, fmaf(zx2, zx2 - 6.f, 3.f), ky * fmaf(xi2, xi2 - 6.f, 3.f));
        const float hxi = -5.770780163555854f * ky * xi * (xi2 - 3.f);
        const float au = fmaf(-2.f, u, fmaf(hxi, cu, -5.770780163555854f * kRoot2G * kx * zx * (zx2 - 3.f)));
        const float av = fmaf(-2.f, v, hxi * cv);
        const float qx = 8.656170245333781f * kRoot2G * kRoot2G * kx * (zx2 - 1.f);
        const float qy = 8.656170245333781f * ky * (xi2 - 1.f), w = fmaf(cu, bx, cv * by);
        const float gx = hx * au, cx = hx * hx * fmaf(qy * cu, cu, 1.f + qx);
        gy = fmaf(bx, au, by * av);
        cy = fmaf(bx * bx, 1.f + qx, fmaf(qy * w, w, by * by));
        A = amp * ex2f(-s) * fmaf(-0.6931471805599453f, e, 1.f + lr);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float d = tile_node(NODES, 7 - i), c = cx * (d * d);
            X[i] = ex2f(fmaf(-gx, d, -c));
            X[7 - i] = ex2f(fmaf(gx, d, -c));
        }
    } else {
        zy = kRoot2G * v;
        gy = -2.f * v * by;
        cy = by * by;
        A = amp * ex2f(-s) * fmaf(-0.6931471805599453f, e, 1.f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float d = tile_node(false, i), a = fmaf(kRoot2G * hx, d, zx), a2 = a * a;
            X[i] = ex2f(-fmaf(2.f * u * hx, d, hx * hx * (d * d))) * fmaf(-r.p[6], fmaf(a2, a2 - 6.f, 3.f), 1.f);
        }
    }
    unsigned rows = 0xffu;  // the tile's rows in the window
    if (!NODES && __any_sync(0xffffffffu, part)) {
        const unsigned cols = window_bits(r.xlo - col0, r.xhi - col0);
        rows = window_bits(r.ylo - row0, r.yhi - row0);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (!(cols >> i & 1u)) X[i] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float d = tile_node(NODES, j);
        float y = A * ex2f(fmaf(gy, d, -(cy * (d * d))));
        if (!COV && !NODES) {
            const float b = fmaf(kRoot2G * by, d, zy), b2 = b * b;
            y *= fmaf(-r.p[7], fmaf(b2, b2 - 6.f, 3.f), 1.f);
        }
        if (!NODES && !(rows >> j & 1u)) y = 0.f;
        const float2 y2 = make_float2(y, y);
        if (COV) {
            const float4 t0 = *reinterpret_cast<const float4 *>(T + 8 * j);
            const float4 t1 = *reinterpret_cast<const float4 *>(T + 8 * j + 4);
            acc[j][0] = __ffma2_rn(make_float2(X[0], X[1]), __fmul2_rn(make_float2(t0.x, t0.y), y2), acc[j][0]);
            acc[j][1] = __ffma2_rn(make_float2(X[2], X[3]), __fmul2_rn(make_float2(t0.z, t0.w), y2), acc[j][1]);
            acc[j][2] = __ffma2_rn(make_float2(X[4], X[5]), __fmul2_rn(make_float2(t1.x, t1.y), y2), acc[j][2]);
            acc[j][3] = __ffma2_rn(make_float2(X[6], X[7]), __fmul2_rn(make_float2(t1.z, t1.w), y2), acc[j][3]);
            asm volatile("" ::: "memory");  // one row's T at a time in registers
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
                acc[j][c] = __ffma2_rn(make_float2(X[2 * c], X[2 * c + 1]), y2, acc[j][c]);
        }
    }
}

// A mid star's tile: the sum over the three y nodes k of X_k[di] Y_k[dj], times T[dj][di] and
// the x correction 1 - kx He4 at the bin's own u (nine operations per bin).
__device__ __forceinline__ void mid_tile(float2 (&acc)[8][4], const StarRec &r,
                                         const float *__restrict__ T, const Tile &tl) {
    const int col0 = tl.col0, row0 = tl.row0;
    const bool over = tl.live && col0 <= r.xhi && col0 + 7 >= r.xlo && row0 <= r.yhi && row0 + 7 >= r.ylo;
    if (!__any_sync(0xffffffffu, over)) return;
    const float hx = r.p[0], bx = r.p[1], by = r.p[2], dn = r.p[7], en = r.p[8];
    const float di0 = over ? (float)col0 + 3.5f - r.ir : 0.f;
    const float dj0 = over ? (float)row0 + 3.5f - r.jr : 0.f;
    const float amp = over ? r.p[3] : 0.f;
    const float u = fmaf(dj0, bx, fmaf(di0, hx, r.p[4])), v = fmaf(dj0, by, r.p[5]);
    // 1 - kx He4(sqrt 2 u / g) = c0 + c1 u^2 + c2 u^4
    const float2 c0 = make_float2(fmaf(-3.f, r.p[6], 1.f), fmaf(-3.f, r.p[6], 1.f));
    const float c1f = 8.317766166719343f * r.p[6], c2f = -1.9218120556728056f * r.p[6];
    const float2 c1 = make_float2(c1f, c1f), c2 = make_float2(c2f, c2f);
    const unsigned cols = window_bits(r.xlo - col0, r.xhi - col0);
    const unsigned rows = window_bits(r.ylo - row0, r.yhi - row0);
    float2 X0[4], Xm[4], Xp[4];
    // u from one pair of columns to the next: its own registers per pair were spilled (k_stamp_tiles of
    // 1,200 templates 2,540 us, 2,420 this way)
    const float2 h0 = make_float2(-3.5f * hx, -2.5f * hx), h2 = make_float2(2.f * hx, 2.f * hx);
    const float hx2 = hx * hx, g0 = -2.f * hx * u, gd = -2.f * hx * dn;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        float x0[2], xm[2], xp[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float d = tile_node(false, 2 * c + q), cx = hx2 * d * d;
            x0[q] = ex2f(fmaf(g0, d, -cx));
            xm[q] = ex2f(fmaf(g0 - gd, d, -cx));
            xp[q] = ex2f(fmaf(g0 + gd, d, -cx));
            if (!(cols >> (2 * c + q) & 1u)) x0[q] = xm[q] = xp[q] = 0.f;
        }
        X0[c] = make_float2(x0[0], x0[1]);
        Xm[c] = make_float2(xm[0], xm[1]);
        Xp[c] = make_float2(xp[0], xp[1]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float d = tile_node(false, j), uj = fmaf(bx, d, u), vj = fmaf(by, d, v);
        const float a = rows >> j & 1u ? amp : 0.f;
        const float um = uj - dn, vm = vj - en, up = uj + dn, vp = vj + en;
        const float y0 = a * ex2f(-fmaf(uj, uj, vj * vj));
        const float ym = 0.625f * a * ex2f(-fmaf(um, um, vm * vm));
        const float yp = 0.625f * a * ex2f(-fmaf(up, up, vp * vp));
        const float2 y02 = make_float2(y0, y0), ym2 = make_float2(ym, ym), yp2 = make_float2(yp, yp);
        float2 uu = __fadd2_rn(make_float2(uj, uj), h0);
        const float4 t0 = *reinterpret_cast<const float4 *>(T + 8 * j);
        const float4 t1 = *reinterpret_cast<const float4 *>(T + 8 * j + 4);
        const float2 t[4] = {make_float2(t0.x, t0.y), make_float2(t0.z, t0.w),
                             make_float2(t1.x, t1.y), make_float2(t1.z, t1.w)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float2 s = __fmul2_rn(uu, uu);
            uu = __fadd2_rn(uu, h2);
            const float2 R = __ffma2_rn(s, __ffma2_rn(s, c2, c1), c0);
            const float2 f = __ffma2_rn(Xp[c], yp2, __ffma2_rn(X0[c], y02, __fmul2_rn(Xm[c], ym2)));
            acc[j][c] = __ffma2_rn(__fmul2_rn(f, t[c]), R, acc[j][c]);
        }
        asm volatile("" ::: "memory");
    }
}

// ---------------------------------------------------------------- the stamp kernels
// A template's smooth (star, strip) pairs on its Chebyshev tiles (k_stamp_nodes), the wide and
// mid stars on its 8 x 8 tiles with the interpolated sums of the smooth pairs added
// (k_stamp_tiles, which writes the template), then the narrow stars (k_stamp_narrow).  Warps
// work by themselves: where the stars lie differs so much from one part of a diagram to the
// next that warps sharing a band in shared memory waited a third of their time for one another.
struct StampStars {
    const double *x, *y, *sx, *sy, *w;
    const StarRec *rec;  // one per star, where the star counts are known to the host
    const int64_t *start;
    const int32_t *count, *cov;
    const StarKey *key = nullptr;  // with rec
};

struct WarpStars {
    StarRec rec[32];  // the warp's current stars
    float T[64];      // and shear table
};

// A warp's walk through a template's stars (first star s0, n of them), of which it takes sg,
// sg + ns, ...: 32 at a time, one per lane, those wanted are compacted into its slots in
// order.  Wanted: wide or mid, with a window that reaches rows ty0 .. ty1; of the wide stars
// those that have (NODES) or lack (else) one of the strips.
// With records the stars are chosen by their keys, fetched 32 ahead (16 bytes a star and one load;
// reading the record's class, rows and strips one after the other waited three times as long).
__device__ __forceinline__ StarKey star_key(const StampStars &st, int64_t s0, int n, int q) {
    if (q >= n) return StarKey{INT_MAX, -1, 0ull};
    const int4 k = __ldg(reinterpret_cast<const int4 *>(st.key + s0 + q));
    return StarKey{k.x, k.y, (unsigned int)k.z | (unsigned long long)(unsigned int)k.w << 32};
}

template <bool NODES, bool REC>
__device__ __forceinline__ int next_stars(StarRec *slot, StarKey &key, const StampStars &st, int64_t s0,
                                          int n, int q0, int sg, int ns, const Grid2 &g, int cov,
                                          int ty0, int ty1, unsigned long long strips) {
    const int lane = threadIdx.x & 31, q = (q0 + lane) * ns + sg;
    StarRec tmp;
    const StarRec *r = &tmp;
    if (REC) {
        r = st.rec + s0 + q;
    } else {
        key = StarKey{INT_MAX, -1, 0ull};
        // (a star whose x step is above 0.1 sqrt 2 sigma is narrow: its FP64 work is not for this kernel)
        if (q < n && 0.70710678f * (float)g.xs / (float)st.sx[s0 + q] <= 0.11f) {
            star_record(tmp, g, st.x[s0 + q], st.y[s0 + q], st.sx[s0 + q], st.sy[s0 + q], st.w[s0 + q], cov);
            if (tmp.cls == kStarWide || tmp.cls == kStarMid) key = StarKey{tmp.ylo, tmp.yhi, 0ull};
        }
    }
    const bool take = key.ylo <= ty1 && key.yhi >= ty0 && ((NODES ? key.strips : ~key.strips) & strips) != 0ull;
    if (REC) key = star_key(st, s0, n, q + 32 * ns);
    const unsigned m = __ballot_sync(0xffffffffu, take);
    if (take) {
        const float4 *from = reinterpret_cast<const float4 *>(r);
        float4 *to = reinterpret_cast<float4 *>(slot + __popc(m & ((1u << lane) - 1u)));
#pragma unroll
        for (int k = 0; k < (int)(sizeof(StarRec) / sizeof(float4)); ++k) to[k] = from[k];
    }
    __syncwarp();
    return __popc(m);
}

// Adds the warp's wide (and mid) stars to the lane's tile.  The warp makes each star's shear
// table, two entries a lane.
template <bool COV, bool NODES, bool REC>
__device__ __forceinline__ void add_stars(float2 (&acc)[8][4], WarpStars &W, const StampStars &st,
                                          int64_t s0, int n, int sg, int ns, const Grid2 &g, int cov,
                                          int ty0, int ty1, unsigned long long strips, const Tile &tl) {
    float *T = W.T;
    // lane: row l / 4 of T, columns 2 (l % 4) and the next; nodes are odd about the middle
    const int lane = threadIdx.x & 31, jr = lane >> 2, jp = jr < 4 ? 3 - jr : jr - 4, ic = lane & 3;
    float tj = jp == 0 ? tile_node(NODES, 4) : jp == 1 ? tile_node(NODES, 5)
               : jp == 2 ? tile_node(NODES, 6) : tile_node(NODES, 7);
    if (jr < 4) tj = -tj;
    if (NODES) tj *= tl.xh * tl.yh;
    const float ti0 = ic == 0 ? tile_node(NODES, 0) : ic == 1 ? tile_node(NODES, 2)
                      : ic == 2 ? tile_node(NODES, 4) : tile_node(NODES, 6);
    const float ti1 = ic == 0 ? tile_node(NODES, 1) : ic == 1 ? tile_node(NODES, 3)
                      : ic == 2 ? tile_node(NODES, 5) : tile_node(NODES, 7);
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[j][c] = make_float2(0.f, 0.f);
    StarKey key{};
    if (REC) key = star_key(st, s0, n, lane * ns + sg);
    for (int q0 = 0; q0 * ns + sg < n; q0 += 32) {
        const int nw = next_stars<NODES, REC>(W.rec, key, st, s0, n, q0, sg, ns, g, cov, ty0, ty1, strips);
#pragma unroll 1
        for (int k = 0; k < nw; ++k) {
            const StarRec &r = W.rec[k];
            if (COV) {
                const float c = -2.f * r.p[0] * r.p[1] * tj;
                const float2 t = make_float2(ex2f(c * ti0), ex2f(c * ti1));
                __syncwarp();  // the previous star's table is no longer read
                *reinterpret_cast<float2 *>(T + 2 * lane) = t;
                __syncwarp();
            }
            if (COV && !NODES && r.cls == kStarMid) mid_tile(acc, r, T, tl);
            else wide_tile<COV, NODES>(acc, r, T, tl);
        }
        __syncwarp();  // the slots are done with
    }
}

// Sums the warps' accumulators in warp order into sum[value][lane] (8 KB).
__device__ __forceinline__ void sum_warps(float *sum, const float2 (&acc)[8][4], int warps) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int w = 0; w < warps; ++w) {
        if (w == warp) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float *v = sum + (8 * j + 2 * c) * 32 + lane;
                    v[0] = w ? v[0] + acc[j][c].x : acc[j][c].x;
                    v[32] = w ? v[32] + acc[j][c].y : acc[j][c].y;
                }
        }
        __syncthreads();
    }
}

// The 8 Chebyshev-node Lagrange weights at x in (-1, 1), nodes ascending:
// (1 + 2 sum_k T_k(c_m) T_k(x)) / 8.
__device__ __forceinline__ void lagrange8(float x, float (&L)[8]) {
    constexpr float c16[9] = {1.f, 0.9807852804032304f, 0.9238795325112867f, 0.8314696123025452f,
                              0.7071067811865476f, 0.5555702330196022f, 0.3826834323650898f,
                              0.19509032201612825f, 0.f};
    float T[8];
    T[0] = 1.f;
    T[1] = x;
#pragma unroll
    for (int k = 2; k < 8; ++k) T[k] = fmaf(2.f * x, T[k - 1], -T[k - 2]);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        float a = 0.125f;
#pragma unroll
        for (int k = 1; k < 8; ++k) {
            const int n = (k * (2 * (7 - m) + 1)) & 31;  // T_k(c_m) = cos(n pi / 16)
            const int f = n <= 16 ? n : 32 - n;
            a = fmaf(0.25f * (f <= 8 ? c16[f] : -c16[16 - f]), T[k], a);
        }
        L[m] = a;
    }
}

// Grid: x -> group of 32 Chebyshev tiles, y -> template; the CTA's warps share the stars.
// node: the tiles' 64 values each, rows of 8.  Most updates come from stars far below the
// detection limit whose errors span the whole diagram (of 5.6e10 updates of the 1,200-template
// build about seven eighths): on these tiles 64 values stand for 640 bins.
__global__ void __launch_bounds__(kNodeWarps * 32, 16 / kNodeWarps)
k_stamp_nodes(StampStars st, Grid2 g0, const Grid2 *__restrict__ grids,
              const int64_t *__restrict__ node_off, int t0, float *__restrict__ node) {
    __shared__ __align__(16) WarpStars W[kNodeWarps];
    __shared__ float sum[2048];
    const int t = t0 + blockIdx.y, group = blockIdx.x;
    const Grid2 g = grids ? grids[t] : g0;
    const Smooth sm = smooth_tiling(g, true);
    if (!sm.on || group >= sm.groups()) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = group * 32 + lane, last = min(group * 32 + 31, sm.tiles() - 1);
    Tile tl{};
    tl.live = tile <= last;
    tl.strip = min(tile, last) / sm.nwc;
    tl.xh = 0.5f * (float)sm.wx;
    tl.yh = 0.5f * (float)sm.wy;
    tl.xc = (float)((tile % sm.nwc) * sm.wx) + tl.xh - 0.5f;
    tl.yc = (float)(tl.strip * sm.wy) + tl.yh - 0.5f;
    const int sa = group * 32 / sm.nwc, sb = last / sm.nwc, cov = st.cov[t];
    float2 acc[8][4];
    if (cov != 0)
        add_stars<true, true, true>(acc, W[warp], st, st.start[t], st.count[t], warp, kNodeWarps, g, cov,
                                    sa * sm.wy, (sb + 1) * sm.wy - 1, strip_bits(sa, sb), tl);
    else
        add_stars<false, true, true>(acc, W[warp], st, st.start[t], st.count[t], warp, kNodeWarps, g, cov,
                                     sa * sm.wy, (sb + 1) * sm.wy - 1, strip_bits(sa, sb), tl);
    sum_warps(sum, acc, kNodeWarps);
    float *out = node + (node_off ? node_off[t] : (int64_t)t * 64 * sm.tiles()) + (int64_t)group * 2048;
    for (int k = threadIdx.x; k < 64 * (last - group * 32 + 1); k += kNodeWarps * 32)
        out[k] = sum[(k & 63) * 32 + (k >> 6)];
}

// One group of 32 tiles of one template per CTA; its ns warps share the stars.  Adds the
// interpolated node values and writes the tiles.
struct StampGroup {
    int32_t t, group;
};

__host__ __device__ inline int tile_groups(int64_t nx, int64_t ny) {
    return (int)((((nx + 7) / 8) * ((ny + 7) / 8) + 31) / 32);
}

template <bool REC>
__global__ void __launch_bounds__(kTileWarpsMax * 32, 1)
k_stamp_tiles(StampStars st, Grid2 g0, int ntempl, const StampGroup *__restrict__ groups,
              const Grid2 *__restrict__ grids, const int64_t *__restrict__ out_off,
              const int64_t *__restrict__ node_off, const float *__restrict__ node,
              float *__restrict__ out) {
    extern __shared__ __align__(16) float smem[];  // [2048] node rows, [ns > 1: 2048] sums, warps
    const int ns = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // on one grid the groups of the last rows first, all templates' together: magnitudes grow with
    // the row, and the faint end's groups take longest
    const StampGroup gr = groups ? groups[blockIdx.x]
                                 : StampGroup{(int)(blockIdx.x % (unsigned)ntempl),
                                              (int)((gridDim.x - 1 - blockIdx.x) / (unsigned)ntempl)};
    const int t = gr.t, cov = st.cov[t];
    const Grid2 g = grids ? grids[t] : g0;
    float *mid = smem, *sum = smem + 2048;
    WarpStars &W = reinterpret_cast<WarpStars *>(smem + (ns > 1 ? 4096 : 2048))[warp];
    const Smooth sm = smooth_tiling(g, node != nullptr);
    const int ntc = (g.nx + 7) >> 3, ntiles = ntc * ((g.ny + 7) >> 3);
    const int tile = gr.group * 32 + lane, last = min(gr.group * 32 + 31, ntiles - 1);
    Tile tl{};
    tl.live = tile <= last;
    tl.col0 = (tile % ntc) * 8;
    tl.row0 = (tile / ntc) * 8;
    tl.strip = tl.live ? tl.row0 / sm.wy : 0;
    const int wa = gr.group * 32 / ntc * 8, wb = min(last / ntc * 8 + 7, g.ny - 1);
    const unsigned long long strips = strip_bits(wa / sm.wy, wb / sm.wy);
    float2 acc[8][4];
    if (cov != 0)
        add_stars<true, false, REC>(acc, W, st, st.start[t], st.count[t], warp, ns, g, cov, wa, wb, strips, tl);
    else
        add_stars<false, false, REC>(acc, W, st, st.start[t], st.count[t], warp, ns, g, cov, wa, wb, strips, tl);
    if (ns > 1) sum_warps(sum, acc, max(1, min(ns, st.count[t])));  // (warps beyond the stars have none)
    if (sm.on) {
        // the tile's 8 columns of its Chebyshev tile's 8 node rows: mid[8 n + i][lane]
        const float *f = node + (node_off ? node_off[t] : (int64_t)t * 64 * sm.tiles()) +
                         64 * (tl.live ? tl.strip * sm.nwc + tl.col0 / sm.wx : 0);
        const float xh = 0.5f * (float)sm.wx;
        for (int i = warp; i < 8; i += ns) {
            float L[8];
            lagrange8(((float)(tl.col0 % sm.wx + i) + 0.5f - xh) / xh, L);
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const float4 a = __ldg(reinterpret_cast<const float4 *>(f + 8 * n));
                const float4 c = __ldg(reinterpret_cast<const float4 *>(f + 8 * n + 4));
                mid[(8 * n + i) * 32 + lane] =
                    fmaf(L[0], a.x, fmaf(L[1], a.y, fmaf(L[2], a.z, fmaf(L[3], a.w,
                    fmaf(L[4], c.x, fmaf(L[5], c.y, fmaf(L[6], c.z, L[7] * c.w)))))));
            }
        }
        if (ns > 1) __syncthreads();
        else __syncwarp();
    }
    if (!tl.live) return;
    float *dst = out + (out_off ? out_off[t] : (int64_t)t * g.nx * g.ny) + (int64_t)tl.row0 * g.nx + tl.col0;
    const bool wide = (g.nx & 3) == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if ((ns > 1 && j % ns != warp) || tl.row0 + j >= g.ny) continue;
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            v[i] = ns > 1 ? sum[(8 * j + i) * 32 + lane] : i & 1 ? acc[j][i >> 1].y : acc[j][i >> 1].x;
        if (sm.on) {
            const float yh = 0.5f * (float)sm.wy;
            float L[8];
            lagrange8(((float)(tl.row0 % sm.wy + j) + 0.5f - yh) / yh, L);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float a = 0.f;
#pragma unroll
                for (int n = 0; n < 8; ++n) a = fmaf(L[n], mid[(8 * n + i) * 32 + lane], a);
                v[i] += a;
            }
        }
        float *row = dst + (int64_t)j * g.nx;
        if (wide) {
            reinterpret_cast<float4 *>(row)[0] = make_float4(v[0], v[1], v[2], v[3]);
            if (tl.col0 + 4 < g.nx) reinterpret_cast<float4 *>(row)[1] = make_float4(v[4], v[5], v[6], v[7]);
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (tl.col0 + i < g.nx) row[i] = v[i];
        }
    }
}

// The narrow stars of all templates (REC: from k_star_prep's list, dealt out star by star; else
// grid y -> template, every star looked at), added to the templates.  Without records a warp makes
// those of its next stars first, a star per lane and as many as leave work for the other warps: a
// record made by one lane holds the FP64 pipe as long as 32.  Calls on 100 x 150 bins, separable narrow
// stars, us, with a record at a time / this way and k_stamp_tiles without their records: 3,000 templates of
// 30 stars 783 / 178, of 100 2,360 / 272, 30 of 3,000 745 / 132, 1 of 30,000 1,044 / 120.
template <bool REC>
__global__ void __launch_bounds__(kNarrowWarps * 32)
k_stamp_narrow(StampStars st, Grid2 g0, const Grid2 *__restrict__ grids,
               const int64_t *__restrict__ out_off, const StarId *__restrict__ narrow,
               const int *__restrict__ n_narrow, int buf, float *__restrict__ out) {
    extern __shared__ float smem[];
    __shared__ __align__(16) StarRec s_rec[kNarrowWarps][REC ? 1 : 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *bx_buf = smem + (size_t)warp * buf, *by_buf = bx_buf + buf - kNarrowRows;
    StarRec *rec = s_rec[warp];
    const int w0 = blockIdx.x * kNarrowWarps + warp, nw = gridDim.x * kNarrowWarps;
    if (REC) {
        const int n = *n_narrow;
        for (int k = w0; k < n; k += nw) {
            const StarId id = narrow[k];
            const Grid2 g = grids ? grids[id.t] : g0;
            const int64_t s = st.start[id.t] + id.q;
            __syncwarp();  // the previous star is done with
            if (lane < (int)(sizeof(StarRec) / 4))
                reinterpret_cast<int *>(rec)[lane] = reinterpret_cast<const int *>(st.rec + s)[lane];
            __syncwarp();
            float *dst = out + (out_off ? out_off[id.t] : (int64_t)id.t * g.nx * g.ny);
            if (rec->cov != 0) star_cov(dst, *rec, g.nx, lane);
            else star_asym(dst, bx_buf, by_buf, *rec, g.nx, lane);
        }
    } else {
        const int t = blockIdx.y, n = st.count[t], cov = st.cov[t];
        const int take = (int)min((int64_t)32, ((int64_t)n + nw - 1) / nw);  // stars of a warp at a time
        const int64_t s0 = st.start[t];
        float *dst = out + (int64_t)t * g0.nx * g0.ny;
        for (int64_t k0 = (int64_t)w0 * take; k0 < n; k0 += (int64_t)nw * take) {
            const int64_t s = s0 + k0 + lane;
            bool mine = false;
            __syncwarp();  // the previous stars are done with
            if (lane < take && k0 + lane < n) {
                star_record(rec[lane], g0, st.x[s], st.y[s], st.sx[s], st.sy[s], st.w[s], cov);
                mine = rec[lane].cls == kStarNarrow;
            }
            const unsigned all = __ballot_sync(0xffffffffu, mine);
            __syncwarp();  // the records are seen by every lane
            for (unsigned m = all; m; m &= m - 1u) {
                const StarRec &r = rec[__ffs(m) - 1];
                if (cov != 0) star_cov(dst, r, g0.nx, lane);
                else star_asym(dst, bx_buf, by_buf, r, g0.nx, lane);
            }
        }
    }
}

__global__ void k_offsets_to_counts(const int64_t *__restrict__ off, int64_t n,
                                    int32_t *__restrict__ cnt) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) cnt[t] = (int32_t)(off[t + 1] - off[t]);
}

// ---------------------------------------------------------------- k_iso_stars (partial_cmd_smooth)
constexpr int kIsoThreads = 256;
constexpr int kIsoMaxPts = 4096;  // isochrone points per template held in shared memory

struct IsoParams {
    int nf, y_index, c1, c2, covariant;
    double dmag;
    // exp_photerr per filter: σ = min(exp2(b (m - c) log2 a) + d, cap)
    double eb_log2a[8], ec[8], ed[8], ecap[8];
    // Martin2016 per filter
    double cA[8], cm50[8], crho_inv[8];
    double bias[8];
    // IMF: segment k covers [lo_k, hi_k) with density scale_k m^-alpha_k / norm
    int nseg;
    double imf_lo[4], imf_hi[4], imf_scale[4], imf_alpha[4];
    double imf_inv_norm, inv_mean_mass;
    int64_t total;  // stride between filters in the mags array
};

struct IsoPoint {
    double mass, xcol, ymag, cerr, yerr, compl_, pdf;
};

// log2 to 2e-9 (the argument of an FP32 exponential, rounded to FP32 after a product with the
// slope): 2^e c_j (1 + r), c_j = 1 + j / 128, |r| < 2^-7, r and log1p(r) in FP32; tab[j] = log c_j.
// The library's FP64 log2 was a sixth of k_iso_stars.
__device__ __forceinline__ double log2_fp32(double x, const sfh_df *__restrict__ tab) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int e = (int)(b >> 52) - 1023, j = (int)(b >> 45) & 127;
    if (e < -1000 || e > 1000) return log2(x);  // negative, subnormal, huge, inf or NaN
    const float c = __uint_as_float(0x3f800000u | (unsigned)j << 16);
    const float r = __fdividef((float)(unsigned)(b >> 13), c) * 1.8189894035458565e-12f;  // 2^-39
    const sfh_df t = tab[j];
    const float l = fmaf(r * r, fmaf(r, fmaf(r, -0.25f, 1.f / 3.f), -0.5f), r);
    return fma((double)t.h + (double)(t.l + l), 1.4426950408889634, (double)e);
}

__device__ __forceinline__ double imf_pdf(const IsoParams &P, double m,
                                          const sfh_df *__restrict__ tab = nullptr) {
    if (!(m >= P.imf_lo[0] && m <= P.imf_hi[P.nseg - 1])) return 0.0;
    int k = 0;
    while (k < P.nseg - 1 && m >= P.imf_hi[k]) ++k;
    return P.imf_scale[k] * P.imf_inv_norm *
           (double)exp2f((float)(-P.imf_alpha[k] * (tab ? log2_fp32(m, tab) : log2(m))));
}

__device__ __forceinline__ double err_eval(const IsoParams &P, int f, double m) {
    const double s = (double)exp2f((float)(P.eb_log2a[f] * (m - P.ec[f]))) + P.ed[f];
    return s < P.ecap[f] ? s : P.ecap[f];
}

__device__ __forceinline__ double compl_eval(const IsoParams &P, int f, double m) {
    return P.cA[f] * rcp_nr(1.0 + (double)__expf((float)((m - P.cm50[f]) * P.crho_inv[f])));
}

// Resampled point q of the isochrone (mini_spacing + interpolate_mini + callables).
__device__ IsoPoint iso_point(const IsoParams &P, const double *m, const double *mags, int n,
                              const int *pos, double dmod, int q) {
    int k = 0;
    double mass, frac;
    if (q == 0) {
        mass = m[0];
        frac = 0.0;
    } else {
        // largest k in [0, n-2] with pos[k] <= q
        int lo = 0, hi = n - 2;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (pos[mid] <= q) lo = mid; else hi = mid - 1;
        }
        k = lo;
        const int j = q - pos[k] + 1;
        const int c = pos[k + 1] - pos[k];
        if (c == 1) {
            mass = m[k + 1];
            frac = 1.0;
        } else {
            frac = (double)j * rcp_nr((double)c);
            mass = fma(m[k + 1] - m[k], frac, m[k]);
        }
    }
    const int kk = (q == 0) ? 0 : k;
    double mag[8];
    int fl[3] = {P.c1, P.c2, P.y_index};
#pragma unroll
    for (int u = 0; u < 3; ++u) {
        const int f = fl[u];
        const double *v = mags + (int64_t)f * P.total;
        const double a = v[kk];
        const double b = (kk + 1 < n) ? v[kk + 1] : a;
        mag[u] = ((q == 0) ? a : a * (1.0 - frac) + b * frac) + dmod;
    }
    IsoPoint p;
    p.mass = mass;
    const double e1 = err_eval(P, P.c1, mag[0]), e2 = err_eval(P, P.c2, mag[1]);
    // (the y filter is usually one of the two)
    const double ey = P.y_index == P.c1 ? e1 : P.y_index == P.c2 ? e2 : err_eval(P, P.y_index, mag[2]);
    double comp = compl_eval(P, P.c1, mag[0]) * compl_eval(P, P.c2, mag[1]);
    if (P.covariant) {
        p.cerr = (P.y_index == P.c1) ? e2 : e1;  // error of the non-y filter, :862
    } else {
        p.cerr = sqrt(e1 * e1 + e2 * e2);        // :871-872
        comp *= compl_eval(P, P.y_index, mag[2]);
    }
    p.yerr = ey;
    p.compl_ = comp;
    p.xcol = (mag[0] + P.bias[P.c1]) - (mag[1] + P.bias[P.c2]);
    p.ymag = mag[2] + P.bias[P.y_index];
    return p;
}

// Segment insertion counts (:128-137) and their exclusive scan: pos[k] is the number of the first
// resampled point of segment k, pos[nseg] = N = 1 + sum(cnt) the number of points.  Flags masses
// that are not strictly increasing (2) and more points than an int counts (1).
__global__ void __launch_bounds__(kIsoThreads)
k_iso_count(const double *__restrict__ m_ini, const double *__restrict__ mags,
            const int64_t *__restrict__ iso_off, const int32_t *__restrict__ iso_len, IsoParams P,
            const double *__restrict__ dmag_t, const int64_t *__restrict__ pos_off,
            int *__restrict__ pos_all, int64_t *__restrict__ nstars_out, int *__restrict__ err_flag) {
    __shared__ int s_warp[2][kIsoThreads / 32];
    const int t = blockIdx.x, nseg = iso_len[t] - 1;
    const double dmag = dmag_t ? dmag_t[t] : P.dmag;
    const double *m = m_ini + iso_off[t], *mg = mags + iso_off[t];
    const double *vc1 = mg + (int64_t)P.c1 * P.total, *vc2 = mg + (int64_t)P.c2 * P.total;
    const double *vy = mg + (int64_t)P.y_index * P.total;
    int *pos = pos_all + pos_off[t];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t carry = 1;
    int round = 0;
    for (int base = 0; base < nseg; base += kIsoThreads, round ^= 1) {
        const int k = base + (int)threadIdx.x;
        int v = 0;
        if (k < nseg) {
            const double dc = (vc1[k + 1] - vc2[k + 1]) - (vc1[k] - vc2[k]);
            const double dy = vy[k + 1] - vy[k];
            const double d = hypot(dc, dy);
            v = 1;
            if (d > dmag) {
                const double r = ceil(d / dmag);
                v = r < 1.0e7 ? (int)r : 10000000;
            }
            if (!(m[k + 1] > m[k])) atomicMax(err_flag, 2);
        }
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_warp[round][warp] = incl;
        __syncthreads();
        int64_t wpre = 0, tot = 0;
        for (int w = 0; w < kIsoThreads / 32; ++w) {
            if (w < warp) wpre += s_warp[round][w];
            tot += s_warp[round][w];
        }
        if (k < nseg) pos[k] = (int)(carry + wpre + incl - v);
        carry += tot;
    }
    if (threadIdx.x == 0) {
        pos[max(nseg, 0)] = (int)carry;
        nstars_out[t] = carry - 1;
        if (carry > INT_MAX) atomicMax(err_flag, 1);
    }
}

// One block of stars: template, first star.
struct IsoBlock {
    int32_t t, base;
};
constexpr int kStarThreads = 128;
constexpr int kIsoStars = kStarThreads - 1;

// A thread per point, blocks of points overlapping by one: a star is a point and its right
// neighbour (midpoints and weight, :765-776, :884-888).  Bound by FP64.  Blocks of 127 stars of any
// template.  With a block per template, which counted the segments over again and took the stars
// in turn, and the y filter's error evaluated a second time: 679 us for 1,200 templates, 684 for
// the 768 of 64 galaxies (0.2 to 5 thousand stars each), 152 for 300, 23 for 6; this way 645, 510,
// 157, 18.
__global__ void __launch_bounds__(kStarThreads)
k_iso_stars(const double *__restrict__ m_ini, const double *__restrict__ mags,
            const int64_t *__restrict__ iso_off, const int32_t *__restrict__ iso_len,
            const double *__restrict__ dmods, const double *__restrict__ norms, IsoParams P,
            const sfh_df *__restrict__ tab, const int64_t *__restrict__ pos_off,
            const int *__restrict__ pos_all, const IsoBlock *__restrict__ blocks, const int64_t *__restrict__ star_off, Grid2 g0,
            const Grid2 *__restrict__ grids, StarRec *__restrict__ rec, StarKey *__restrict__ key,
            StarId *__restrict__ narrow, int *__restrict__ n_narrow) {
    __shared__ IsoPoint s_pt[kStarThreads];
    __shared__ int s_pos[kIsoMaxPts];
    const IsoBlock blk = blocks[blockIdx.x];
    const int t = blk.t, n = iso_len[t];
    const int *pos = pos_all + pos_off[t];
    for (int k = threadIdx.x; k < n; k += kStarThreads) s_pos[k] = pos[k];
    __syncthreads();
    const double *m = m_ini + iso_off[t], *mg = mags + iso_off[t];
    const int npts = s_pos[n - 1];
    const int64_t so = star_off[t];
    const Grid2 g = grids ? grids[t] : g0;
    const int cov = P.covariant ? (P.y_index == P.c1 ? -1 : 1) : 0;
    const int q = blk.base + (int)threadIdx.x;
    IsoPoint a;
    if (q < npts) {
        a = iso_point(P, m, mg, n, s_pos, dmods[t], q);
        a.pdf = imf_pdf(P, a.mass, tab);
        s_pt[threadIdx.x] = a;
    }
    __syncthreads();
    if (threadIdx.x < kIsoStars && q < npts - 1) {
        const IsoPoint &b = s_pt[threadIdx.x + 1];
        const double wscale = norms[t] * P.inv_mean_mass;
        const double w = (b.mass - a.mass) * (a.pdf + b.pdf) * 0.5 * a.compl_ * wscale;
        StarRec r{};
        star_record(r, g, a.xcol + (b.xcol - a.xcol) * 0.5, a.ymag + (b.ymag - a.ymag) * 0.5,
                    a.cerr + (b.cerr - a.cerr) * 0.5, a.yerr + (b.yerr - a.yerr) * 0.5, w, cov);
        store_record(r, g, StarId{t, q}, rec + so + q, key + so + q, narrow, n_narrow);
    }
}

// The widest accepted grid: a separable narrow star's x table of four warps in shared memory.
constexpr int64_t kMaxColumns = 3123;

// Warps per tile group: as many as the stars can be dealt to while all groups together stay
// within six waves of 16 warps (128 registers) per SM: a group in the dense part of a diagram takes
// several times the mean, and one warp of it would be the tail.  Templates on grids of their own
// have different numbers of stars too: four times that.  k_stamp_tiles with 1, 2, 4, 8, 16 warps,
// us: 60 binary templates (1,800 groups) 1,500, -, 335, 292, 394; 300 separable (5,100) 173, 180,
// 201, 295; 1,200 (36,000) 2,420 with one; 768 templates of 64 galaxies (12,360) 1,880, 1,500, 1,360.
// No more than a template has stars (the warps' sums are added one after the other), as the narrow
// stars' blocks are no more than there can be stars for: one star on 200 x 300 bins 120 us a call without these
// two limits, 116 with.
int tile_warps(int64_t groups, bool uneven, int64_t maxcount, int sm_count) {
    const int64_t most = (uneven ? 384 : 96) * (int64_t)sm_count;
    int ns = 1;
    while (ns < kTileWarpsMax && ns < maxcount && groups * 2 * ns <= most) ns *= 2;
    return ns;
}

int check_grid(sfh_ctx *ctx, int64_t nx, int64_t ny) {
    if (nx < 1 || ny < 1 || nx > (1 << 20) || ny > (1 << 20))
        return sfh_set_error(ctx, SFH_ERR_ARG, "stamp grid or template count out of range");
    if (nx > kMaxColumns)
        return sfh_set_error(ctx, SFH_ERR_UNSUPPORTED, "Hess grid too wide for a shared-memory band");
    return SFH_OK;
}

size_t tile_smem(int ns) { return (ns > 1 ? 16384 : 8192) + ns * sizeof(WarpStars); }

// Bytes of the node values of ntempl templates on one grid.
size_t node_bytes(const Grid2 &g, int64_t ntempl) {
    const Smooth sm = smooth_tiling(g, true);
    return sm.on ? (size_t)ntempl * 64 * sm.tiles() * sizeof(float) : 0;
}

// Device workspace of the stamps, where the star counts are known to the host.
struct StampWork {
    StarRec *rec = nullptr;    // one per star, indexed as the star arrays
    StarKey *key = nullptr;    // the same
    StarId *narrow = nullptr;  // room for every star
    int *n_narrow = nullptr;
    float *node = nullptr;     // node_bytes() / the ragged batch's nodes
    int64_t stars = 0, maxcount = 0;  // of all templates, of the one with the most
    bool made = false;         // the records are there already (k_iso_stars)
    bool smooth = true;        // Chebyshev tiles are used (made records always expect them)
    static size_t bytes(int64_t stars, size_t node) {
        const size_t n = (size_t)std::max<int64_t>(stars, 1);
        return 256 + sfh_align256(n * sizeof(StarRec)) + sfh_align256(n * sizeof(StarKey)) +
               sfh_align256(n * sizeof(StarId)) + sfh_align256(node);
    }
    StampWork() = default;
    StampWork(char *b, int64_t stars_, int64_t maxcount_) : stars(stars_), maxcount(maxcount_) {
        const size_t n = (size_t)std::max<int64_t>(stars, 1);
        n_narrow = (int *)b;
        rec = (StarRec *)(b += 256);
        key = (StarKey *)(b += sfh_align256(n * sizeof(StarRec)));
        narrow = (StarId *)(b += sfh_align256(n * sizeof(StarKey)));
        node = (float *)(b + sfh_align256(n * sizeof(StarId)));
    }
};

// bin_cmd_smooth of fewer stars does without the Chebyshev tiles: a launch and the interpolation cost
// more than they save.  200 x 300 bins, 1, 10, 30 separable stars of 0.2 bins' error, call in us: 116,
// 116, 118 with, 100, 109, 110 without (a block per band of rows, as once, 108, 116, 121); covariant
// stars of 30 bins' error 116, 118, 121 with, 100, 106, 115 without.
constexpr int kSmoothStars = 64;

// Per-template grids of a ragged batch on the device.
struct StampGrids {
    const Grid2 *grids;
    const int64_t *out_off, *node_off;
    const StampGroup *groups;
    int64_t ngroups;
    int max_node_groups;
    int64_t max_nx;
};

// Stamps of ntempl templates, on one grid g or (rg) each on its own.  Without work->rec (the
// caller does not know the star counts) every kernel makes the records it needs and no strips
// are smooth.
int launch_stamps(sfh_ctx *ctx, StampStars st, int64_t ntempl, Grid2 g, const StampGrids *rg,
                  const StampWork &w, float *d_out) {
    const int64_t nx = rg ? rg->max_nx : g.nx;
    if (!rg && (ntempl < 1 || ntempl > 65535))
        return sfh_set_error(ctx, SFH_ERR_ARG, "stamp grid or template count out of range");
    if (int rc = rg ? SFH_OK : check_grid(ctx, nx, g.ny)) return rc;
    const bool have = w.rec != nullptr;
    st.rec = w.rec;
    st.key = w.key;
    const Smooth sm = smooth_tiling(g, have && !rg && w.smooth);
    const int node_groups = rg ? rg->max_node_groups : sm.on ? sm.groups() : 0;
    cudaStream_t s = ctx->stream;
    if (have && !w.made) SFH_CK(ctx, cudaMemsetAsync(w.n_narrow, 0, sizeof(int), s));
    for (int64_t t0 = 0; have && t0 < ntempl; t0 += 65535) {
        const unsigned nt = (unsigned)std::min<int64_t>(65535, ntempl - t0);
        if (w.maxcount > 0 && !w.made) {
            k_star_prep<<<dim3((unsigned)((w.maxcount + kPrepThreads - 1) / kPrepThreads), nt),
                          kPrepThreads, 0, s>>>(st.x, st.y, st.sx, st.sy, st.w, st.start, st.count,
                                                st.cov, g, rg ? rg->grids : nullptr, (int)t0, w.smooth,
                                                w.rec, w.key, w.narrow, w.n_narrow);
            SFH_LAUNCHED(ctx);
        }
        if (node_groups > 0) {
            k_stamp_nodes<<<dim3((unsigned)node_groups, nt), kNodeWarps * 32, 0, s>>>(
                st, g, rg ? rg->grids : nullptr, rg ? rg->node_off : nullptr, (int)t0, w.node);
            SFH_LAUNCHED(ctx);
        }
    }
    const int64_t groups = rg ? rg->ngroups : ntempl * tile_groups(g.nx, g.ny);
    const int ns = tile_warps(groups, rg != nullptr, have ? w.maxcount : INT_MAX, ctx->sm_count);
    auto tiles = have ? k_stamp_tiles<true> : k_stamp_tiles<false>;
    // (raised at every launch: a limit belongs to the device; always the most, for all threads)
    if (tile_smem(ns) > 48 * 1024)
        SFH_CK(ctx, cudaFuncSetAttribute(tiles, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)tile_smem(kTileWarpsMax)));
    tiles<<<(unsigned)groups, 32 * ns, tile_smem(ns), s>>>(
        st, g, (int)ntempl, rg ? rg->groups : nullptr, rg ? rg->grids : nullptr, rg ? rg->out_off : nullptr,
        rg ? rg->node_off : nullptr, node_groups > 0 ? w.node : nullptr, d_out);
    SFH_LAUNCHED(ctx);
    const int buf = (int)nx + kNarrowRows;
    // Eight times the blocks that are resident (7 per SM, by registers), so that the last wave is a
    // small part and the stars' sizes even out: 1,200 templates 696 us with eight blocks per SM (the
    // eighth alone in a second wave), 610 with 7, 529 with 56, 515 with 112; 300 separable ones 230,
    // 202, 164, 162; 6 small ones 13 with any.
    // Without records twice the resident ones: a warp takes up to 32 stars at a time there.
    const unsigned blocks = 56u * (unsigned)ctx->sm_count;
    const dim3 ngrid = have ? dim3((unsigned)std::clamp<int64_t>((w.stars + kNarrowWarps - 1) / kNarrowWarps, 1, blocks))
                            : dim3(std::max(1u, 14u * (unsigned)ctx->sm_count / (unsigned)ntempl), (unsigned)ntempl);
    auto narrow = have ? k_stamp_narrow<true> : k_stamp_narrow<false>;
    const size_t nsmem = kNarrowWarps * (size_t)buf * sizeof(float);
    if (nsmem > 36 * 1024)  // (beside the records)
        SFH_CK(ctx, cudaFuncSetAttribute(narrow, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(kNarrowWarps * (kMaxColumns + kNarrowRows) * sizeof(float))));
    narrow<<<ngrid, kNarrowWarps * 32, nsmem, s>>>(
        st, g, rg ? rg->grids : nullptr, rg ? rg->out_off : nullptr, w.narrow, w.n_narrow, buf, d_out);
    SFH_LAUNCHED(ctx);
    return SFH_OK;
}

}  // namespace

extern "C" int sfh_bin_cmd_smooth_batch_dev(sfh_ctx *ctx, const double *d_x, const double *d_y,
                                            const double *d_sx, const double *d_sy,
                                            const double *d_w, const int64_t *d_offsets,
                                            const int32_t *h_cov, int64_t ntempl, double xf,
                                            double xs, int64_t nx, double yf, double ys,
                                            int64_t ny, float *d_models) {
    if (!ctx || !d_x || !d_y || !d_sx || !d_sy || !d_w || !d_offsets || !h_cov || !d_models ||
        ntempl < 1)
        return SFH_ERR_ARG;
    for (int64_t t = 0; t < ntempl; ++t)
        if (h_cov[t] < -1 || h_cov[t] > 1) return sfh_set_error(ctx, SFH_ERR_ARG, "cov_mult must be -1, 0 or 1");
    SFH_CK(ctx, cudaSetDevice(ctx->device));
    const size_t o_cnt = 0, o_cov = sfh_align256(ntempl * 4);
    int rc = sfh_scratch_reserve(ctx, o_cov + sfh_align256(ntempl * 4));
    if (rc) return rc;
    int32_t *d_cnt = (int32_t *)((char *)ctx->scratch + o_cnt);
    int32_t *d_cov = (int32_t *)((char *)ctx->scratch + o_cov);
    SFH_CK(ctx, cudaMemcpyAsync(d_cov, h_cov, ntempl * 4, cudaMemcpyHostToDevice, ctx->stream));
    k_offsets_to_counts<<<(int)((ntempl + 255) / 256), 256, 0, ctx->stream>>>(d_offsets, ntempl,
                                                                                d_cnt);
    SFH_LAUNCHED(ctx);
    const Grid2 g = make_grid(xf, xs, nx, yf, ys, ny);
    return launch_stamps(ctx, StampStars{d_x, d_y, d_sx, d_sy, d_w, nullptr, d_offsets, d_cnt, d_cov},
                         ntempl, g, nullptr, StampWork(), d_models);
}

extern "C" int sfh_bin_cmd_smooth(sfh_ctx *ctx, const double *x, const double *y,
                                  const double *sx, const double *sy, const double *w,
                                  int64_t npts, int cov_mult, double xf, double xs, int64_t nx,
                                  double yf, double ys, int64_t ny, double *hist_out) {
    if (!ctx || !hist_out || npts < 0 || nx < 1 || ny < 1) return SFH_ERR_ARG;
    if (npts > 0 && (!x || !y || !sx || !sy || !w)) return SFH_ERR_ARG;
    if (cov_mult < -1 || cov_mult > 1)  // @argcheck cov_mult in (-1, 0, 1), :578
        return sfh_set_error(ctx, SFH_ERR_ARG, "cov_mult must be -1, 0 or 1");
    for (int64_t i = 0; i < npts; ++i)
        if (sx[i] < 0.0 || sy[i] < 0.0)
            return sfh_set_error(ctx, SFH_ERR_ARG, "photometric errors must be non-negative");
    SFH_CK(ctx, cudaSetDevice(ctx->device));
    const int64_t nbins = nx * ny;
    const size_t a5 = sfh_align256((size_t)(npts > 0 ? npts : 1) * 8);
    const size_t o_out = 5 * a5, o_meta = o_out + sfh_align256(nbins * 4), o_work = o_meta + 256;
    if (nx > (1 << 20) || ny > (1 << 20))
        return sfh_set_error(ctx, SFH_ERR_ARG, "stamp grid or template count out of range");
    const Grid2 g = make_grid(xf, xs, nx, yf, ys, ny);
    int rc = sfh_stage_reserve(ctx, o_work + StampWork::bytes(npts, node_bytes(g, 1)));
    if (rc) return rc;
    char *b = (char *)ctx->stage;
    const double *src[5] = {x, y, sx, sy, w};
    for (int k = 0; k < 5 && npts > 0; ++k)
        SFH_CK(ctx, cudaMemcpyAsync(b + k * a5, src[k], npts * 8, cudaMemcpyHostToDevice, ctx->stream));
    struct { int64_t start; int32_t count; int32_t cov; } meta{0, (int32_t)npts, cov_mult};
    SFH_CK(ctx, cudaMemcpyAsync(b + o_meta, &meta, sizeof(meta), cudaMemcpyHostToDevice, ctx->stream));
    float *d_out = (float *)(b + o_out);
    StampWork work(b + o_work, npts, npts);
    work.smooth = npts >= kSmoothStars;
    rc = launch_stamps(ctx, StampStars{(const double *)b, (const double *)(b + a5),
                                       (const double *)(b + 2 * a5), (const double *)(b + 3 * a5),
                                       (const double *)(b + 4 * a5), nullptr,
                                       (const int64_t *)(b + o_meta), (const int32_t *)(b + o_meta + 8),
                                       (const int32_t *)(b + o_meta + 12)},
                       1, g, nullptr, work, d_out);
    if (rc) return rc;
    std::vector<float> tmp((size_t)nbins);
    SFH_CK(ctx, cudaMemcpyAsync(tmp.data(), d_out, nbins * 4, cudaMemcpyDeviceToHost, ctx->stream));
    SFH_CK(ctx, cudaStreamSynchronize(ctx->stream));
    for (int64_t i = 0; i < nbins; ++i) hist_out[i] = tmp[(size_t)i];
    return SFH_OK;
}

namespace {
// Validates the filter indices, IMF and callables of partial_cmd_smooth and fills the
// device-side parameter block (everything but the grid-dependent Δmag).
int make_iso_params(sfh_ctx *ctx, int nf, int y_index, int c1, int c2, const sfh_err_model *err,
                    const sfh_compl_model *compl_, const double *bias, const sfh_imf *imf,
                    double mean_mass, int64_t total, IsoParams &P) {
    if (nf < 2 || nf > 8 || y_index < 0 || y_index >= nf || c1 < 0 || c1 >= nf || c2 < 0 ||
        c2 >= nf || c1 == c2)
        return sfh_set_error(ctx, SFH_ERR_ARG, "invalid filter indices");
    if (imf->nseg < 1 || imf->nseg > 4 || !(imf->mmin > 0) || !(imf->mmax > imf->mmin) ||
        !(mean_mass > 0))
        return sfh_set_error(ctx, SFH_ERR_ARG, "invalid IMF");
    P = IsoParams{};
    P.nf = nf;
    P.y_index = y_index;
    P.c1 = c1;
    P.c2 = c2;
    P.covariant = (y_index == c1 || y_index == c2) ? 1 : 0;
    P.total = total;
    for (int f = 0; f < nf; ++f) {
        if (!(err[f].a > 0) || !(compl_[f].rho != 0))
            return sfh_set_error(ctx, SFH_ERR_ARG, "invalid error or completeness model");
        P.eb_log2a[f] = err[f].b * std::log2(err[f].a);
        P.ec[f] = err[f].c;
        P.ed[f] = err[f].d;
        P.ecap[f] = err[f].cap;
        P.cA[f] = compl_[f].A;
        P.cm50[f] = compl_[f].m50;
        P.crho_inv[f] = 1.0 / compl_[f].rho;
        P.bias[f] = bias ? bias[f] : 0.0;
    }
    // IMF segments: continuity at the breaks, normalised on [mmin, mmax].
    P.nseg = imf->nseg;
    double s = 1.0, norm = 0.0;
    for (int k = 0; k < imf->nseg; ++k) {
        const double lo = (k == 0) ? imf->mmin : imf->breaks[k - 1];
        const double hi = (k == imf->nseg - 1) ? imf->mmax : imf->breaks[k];
        if (k > 0) s *= std::pow(lo, imf->alpha[k] - imf->alpha[k - 1]);
        P.imf_lo[k] = lo;
        P.imf_hi[k] = hi;
        P.imf_scale[k] = s;
        P.imf_alpha[k] = imf->alpha[k];
        const double p = 1.0 - imf->alpha[k];
        norm += s * (std::fabs(p) < 1e-14 ? std::log(hi / lo) : (std::pow(hi, p) - std::pow(lo, p)) / p);
    }
    P.imf_inv_norm = 1.0 / norm;
    P.inv_mean_mass = 1.0 / mean_mass;
    return SFH_OK;
}

// Isochrone lengths and offsets inside the concatenated point arrays.
int check_isochrones(sfh_ctx *ctx, const int64_t *h_iso_off, const int32_t *h_iso_len,
                     int64_t ntempl, int64_t total) {
    for (int64_t t = 0; t < ntempl; ++t) {
        const int32_t n = h_iso_len[t];
        if (n < 2 || n > kIsoMaxPts)
            return sfh_set_error(ctx, SFH_ERR_ARG, "isochrone length must be in [2, 4096]");
        if (h_iso_off[t] < 0 || h_iso_off[t] + n > total)
            return sfh_set_error(ctx, SFH_ERR_ARG, "isochrone offsets out of range");
    }
    return SFH_OK;
}
}  // namespace

namespace {
// Host-side description of per-template Hess grids (ragged galaxies).
struct RaggedSpec {
    std::vector<Grid2> grids;
    std::vector<int64_t> out_off, node_off;
    int64_t nodes = 0;   // node values of all templates
    int max_node_groups = 0;  // largest template's groups of 32 Chebyshev tiles
    std::vector<double> dmag;
    std::vector<StampGroup> groups;  // every template's groups of 32 tiles
    int64_t max_nx = 0;
};

// The two device passes of partial_cmd_smooth for a batch of isochrones (resampled star
// counts, then star records), followed by the stamps on one shared grid (rg == nullptr)
// or on each template's own grid.
int partial_run(sfh_ctx *ctx, const double *d_m_ini, const double *d_mags,
                const int64_t *h_iso_off, const int32_t *h_iso_len, int64_t ntempl,
                const IsoParams &P, int y_index, int c1, const double *h_dmod,
                const double *h_norm, const RaggedSpec *rg, double xf, double xs, int64_t nx,
                double yf, double ys, int64_t ny, float *d_models) {
    cudaStream_t st = ctx->stream;
    // What the host knows, in one upload, ending in the zeroed counters; the star counts follow
    // them, so that pass 1 is read back in one copy.
    std::vector<char> head;
    auto add = [](std::vector<char> &to, const void *src, size_t bytes) {
        const size_t at = to.size();
        to.resize(at + sfh_align256(bytes), 0);
        if (src) std::memcpy(to.data() + at, src, bytes);
        return at;
    };
    const size_t n8 = (size_t)ntempl * 8, n4 = (size_t)ntempl * 4;
    const std::vector<int32_t> cov((size_t)ntempl, P.covariant ? (y_index == c1 ? -1 : 1) : 0);
    std::vector<int64_t> poff((size_t)ntempl);
    int64_t npos = 0;
    for (int64_t t = 0; t < ntempl; ++t) {
        poff[(size_t)t] = npos;
        npos += std::max(h_iso_len[t], 1);
    }
    const size_t o_off = add(head, h_iso_off, n8), o_len = add(head, h_iso_len, n4);
    const size_t o_dm = add(head, h_dmod, n8), o_nm = add(head, h_norm, n8);
    const size_t o_cov = add(head, cov.data(), n4), o_poff = add(head, poff.data(), n8);
    const size_t o_dmag = rg ? add(head, rg->dmag.data(), n8) : 0;
    const size_t o_grid = rg ? add(head, rg->grids.data(), ntempl * sizeof(Grid2)) : 0;
    const size_t o_oof = rg ? add(head, rg->out_off.data(), n8) : 0;
    const size_t o_noff = rg ? add(head, rg->node_off.data(), n8) : 0;
    const size_t o_groups = rg ? add(head, rg->groups.data(), rg->groups.size() * sizeof(StampGroup)) : 0;
    const size_t o_err = add(head, nullptr, 8), o_cnt64 = head.size();  // error flag, narrow stars
    const size_t o_pos = o_cnt64 + sfh_align256(n8), o_late = o_pos + sfh_align256((size_t)npos * 4);
    // Pass 1: resampled star count per template (one read-back), exact offsets.
    int rc = sfh_scratch_reserve(ctx, o_late);
    if (rc) return rc;
    char *b = (char *)ctx->scratch;
    const auto dmag = [&] { return rg ? (const double *)(b + o_dmag) : nullptr; };  // per-template Δmag
    const auto pass1 = [&]() -> int {
        SFH_CK(ctx, cudaMemcpyAsync(b, head.data(), head.size(), cudaMemcpyHostToDevice, st));
        k_iso_count<<<(unsigned)ntempl, kIsoThreads, 0, st>>>(
            d_m_ini, d_mags, (const int64_t *)(b + o_off), (const int32_t *)(b + o_len), P, dmag(),
            (const int64_t *)(b + o_poff), (int *)(b + o_pos), (int64_t *)(b + o_cnt64), (int *)(b + o_err));
        SFH_LAUNCHED(ctx);
        return SFH_OK;
    };
    if ((rc = pass1())) return rc;
    std::vector<int64_t> back((o_cnt64 - o_err) / 8 + (size_t)ntempl);
    SFH_CK(ctx, cudaMemcpyAsync(back.data(), b + o_err, back.size() * 8, cudaMemcpyDeviceToHost, st));
    SFH_CK(ctx, cudaStreamSynchronize(st));
    int flag = 0;
    std::memcpy(&flag, back.data(), 4);
    if (flag == 2) return sfh_set_error(ctx, SFH_ERR_ARG, "isochrone masses must be strictly increasing");
    if (!rg && (rc = check_grid(ctx, nx, ny))) return rc;  // (a ragged batch's grids were checked)
    if (flag == 1) return sfh_set_error(ctx, SFH_ERR_NOMEM, "too many resampled points in an isochrone");
    const int64_t *nst = back.data() + (o_cnt64 - o_err) / 8;
    std::vector<int64_t> soff((size_t)ntempl + 1);
    std::vector<int32_t> count((size_t)ntempl);
    int64_t maxcount = 0, nblocks = 0;
    for (int64_t t = 0; t < ntempl; ++t) {
        soff[(size_t)t + 1] = soff[(size_t)t] + nst[t];
        count[(size_t)t] = (int32_t)nst[t];
        maxcount = std::max(maxcount, nst[t]);
        nblocks += (nst[t] + kIsoStars - 1) / kIsoStars;
    }
    const int64_t nstar_total = std::max<int64_t>(soff[(size_t)ntempl], 1);
    const size_t late_bytes = sfh_align256(n8 + 8) + sfh_align256(n4) +
                              sfh_align256((size_t)nblocks * sizeof(IsoBlock));
    const size_t o_work = o_late + late_bytes;
    // Pass 2: star records, then the stamps.
    const Grid2 g = make_grid(xf, xs, nx, yf, ys, ny);
    const size_t nodes = rg ? (size_t)rg->nodes * sizeof(float) : node_bytes(g, ntempl);
    const size_t had = ctx->scratch_bytes;
    rc = sfh_scratch_reserve(ctx, o_work + StampWork::bytes(nstar_total, nodes));
    if (rc) return rc;
    if (ctx->scratch_bytes != had) {  // a new scratch, perhaps at the old address: pass 1's results anew
        b = (char *)ctx->scratch;
        if ((rc = pass1())) return rc;
    }
    std::vector<IsoBlock> blocks;
    blocks.reserve((size_t)nblocks);
    for (int64_t t = 0; t < ntempl; ++t)
        for (int64_t q = 0; q < nst[t]; q += kIsoStars) blocks.push_back(IsoBlock{(int32_t)t, (int32_t)q});
    std::vector<char> late;  // known after pass 1
    late.reserve(late_bytes);
    const size_t o_soff = o_late + add(late, soff.data(), n8 + 8), o_cnt = o_late + add(late, count.data(), n4);
    const size_t o_blk = o_late + add(late, blocks.data(), blocks.size() * sizeof(IsoBlock));
    SFH_CK(ctx, cudaMemcpyAsync(b + o_late, late.data(), late.size(), cudaMemcpyHostToDevice, st));
    StampWork work(b + o_work, nstar_total, maxcount);
    work.made = true;
    work.n_narrow = (int *)(b + o_err) + 1;
    if (nblocks > 0) {
        k_iso_stars<<<(unsigned)nblocks, kStarThreads, 0, st>>>(
            d_m_ini, d_mags, (const int64_t *)(b + o_off), (const int32_t *)(b + o_len),
            (const double *)(b + o_dm), (const double *)(b + o_nm), P, ctx->d_df_tab,
            (const int64_t *)(b + o_poff),
            (const int *)(b + o_pos), (const IsoBlock *)(b + o_blk), (const int64_t *)(b + o_soff), g,
            rg ? (const Grid2 *)(b + o_grid) : nullptr, work.rec, work.key, work.narrow, work.n_narrow);
        SFH_LAUNCHED(ctx);
    }
    StampGrids sg{};
    if (rg)
        sg = StampGrids{(const Grid2 *)(b + o_grid), (const int64_t *)(b + o_oof),
                        (const int64_t *)(b + o_noff), (const StampGroup *)(b + o_groups),
                        (int64_t)rg->groups.size(), rg->max_node_groups, rg->max_nx};
    rc = launch_stamps(ctx, StampStars{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                                       (const int64_t *)(b + o_soff), (const int32_t *)(b + o_cnt),
                                       (const int32_t *)(b + o_cov)},
                       ntempl, g, rg ? &sg : nullptr, work, d_models);
    if (rc) return rc;
    SFH_CK(ctx, cudaStreamSynchronize(st));
    return SFH_OK;
}
}  // namespace

extern "C" int sfh_partial_cmd_smooth_batch_dev(
    sfh_ctx *ctx, const double *d_m_ini, const double *d_mags, int64_t total,
    const int64_t *h_iso_off, const int32_t *h_iso_len, int64_t ntempl, int nf, int y_index,
    int c1, int c2, const sfh_err_model *err, const sfh_compl_model *compl_, const double *bias,
    const sfh_imf *imf, double mean_mass, const double *h_dmod, const double *h_norm, double xf,
    double xs, int64_t nx, double yf, double ys, int64_t ny, float *d_models) {
    if (!ctx || !d_m_ini || !d_mags || !h_iso_off || !h_iso_len || !err || !compl_ || !imf ||
        !h_dmod || !h_norm || !d_models || ntempl < 1 || ntempl > 65535)
        return SFH_ERR_ARG;
    SFH_CK(ctx, cudaSetDevice(ctx->device));
    IsoParams P;
    int rc0 = make_iso_params(ctx, nf, y_index, c1, c2, err, compl_, bias, imf, mean_mass, total, P);
    if (rc0) return rc0;
    P.dmag = std::fmin(std::fabs(xs), std::fabs(ys));  // :851
    if ((rc0 = check_isochrones(ctx, h_iso_off, h_iso_len, ntempl, total))) return rc0;
    return partial_run(ctx, d_m_ini, d_mags, h_iso_off, h_iso_len, ntempl, P, y_index, c1, h_dmod,
                       h_norm, nullptr, xf, xs, nx, yf, ys, ny, d_models);
}

extern "C" int sfh_partial_cmd_smooth_ragged_dev(
    sfh_ctx *ctx, const double *d_m_ini, const double *d_mags, int64_t total,
    const int64_t *h_iso_off, const int32_t *h_iso_len, int64_t ntempl, int nf, int y_index,
    int c1, int c2, const sfh_err_model *err, const sfh_compl_model *compl_, const double *bias,
    const sfh_imf *imf, double mean_mass, const double *h_dmod, const double *h_norm,
    const sfh_hess_grid *h_grids, int64_t models_len, float *d_models) {
    if (!ctx || !d_m_ini || !d_mags || !h_iso_off || !h_iso_len || !err || !compl_ || !imf ||
        !h_dmod || !h_norm || !h_grids || !d_models || ntempl < 1 || ntempl > (1 << 24) ||
        models_len < 1)
        return SFH_ERR_ARG;
    SFH_CK(ctx, cudaSetDevice(ctx->device));
    IsoParams P;
    int rc0 = make_iso_params(ctx, nf, y_index, c1, c2, err, compl_, bias, imf, mean_mass, total, P);
    if (rc0) return rc0;
    if ((rc0 = check_isochrones(ctx, h_iso_off, h_iso_len, ntempl, total))) return rc0;
    RaggedSpec rg;
    rg.grids.resize((size_t)ntempl);
    rg.out_off.resize((size_t)ntempl);
    rg.node_off.resize((size_t)ntempl);
    rg.dmag.resize((size_t)ntempl);
    int64_t ngroups = 0;
    for (int64_t t = 0; t < ntempl; ++t) {
        const sfh_hess_grid &h = h_grids[t];
        if (h.nx < 1 || h.ny < 1 || h.nx > (1 << 20) || h.ny > (1 << 20) || !(h.x_step != 0) ||
            !(h.y_step != 0))
            return sfh_set_error(ctx, SFH_ERR_ARG, "Hess grid out of range");
        if (h.out_offset < 0 || h.out_offset + h.nx * h.ny > models_len)
            return sfh_set_error(ctx, SFH_ERR_ARG, "template output outside d_models");
        if (h.nx > kMaxColumns)
            return sfh_set_error(ctx, SFH_ERR_UNSUPPORTED, "Hess grid too wide for a shared-memory band");
        rg.grids[(size_t)t] = make_grid(h.x_first, h.x_step, h.nx, h.y_first, h.y_step, h.ny);
        rg.out_off[(size_t)t] = h.out_offset;
        rg.node_off[(size_t)t] = rg.nodes;
        const Smooth sm = smooth_tiling(rg.grids[(size_t)t], true);
        if (sm.on) {
            rg.nodes += 64 * (int64_t)sm.tiles();
            rg.max_node_groups = std::max(rg.max_node_groups, sm.groups());
        }
        rg.dmag[(size_t)t] = std::fmin(std::fabs(h.x_step), std::fabs(h.y_step));  // :851
        rg.max_nx = std::max(rg.max_nx, h.nx);
        ngroups += tile_groups(h.nx, h.ny);
    }
    if (ngroups > 0x7fffffff) return sfh_set_error(ctx, SFH_ERR_UNSUPPORTED, "too many stamp tiles");
    // the last rows of every grid first, as on one grid
    rg.groups.reserve((size_t)ngroups);
    constexpr int kBands = 16;
    for (int q = kBands - 1; q >= 0; --q)
        for (int64_t t = 0; t < ntempl; ++t) {
            const int64_t n = tile_groups(rg.grids[(size_t)t].nx, rg.grids[(size_t)t].ny);
            for (int64_t k = n * q / kBands; k < n * (q + 1) / kBands; ++k)
                rg.groups.push_back(StampGroup{(int32_t)t, (int32_t)k});
        }
    P.dmag = rg.dmag[0];
    return partial_run(ctx, d_m_ini, d_mags, h_iso_off, h_iso_len, ntempl, P, y_index, c1, h_dmod,
                       h_norm, &rg, 0.0, 0.0, 0, 0.0, 0.0, 0, d_models);
}

// ---------------------------------------------------------------- binary_hess (RandomBinaryPairs)
// src/StarFormationHistories.jl:627-706 for a batch of templates: every pair (i, j > i) of
// interval left points of a template's (downsampled) isochrone is a binary system whose
// magnitudes add in flux (:656), weighted ΔMp ΔMs (imf_i + imf_i+1)(imf_j + imf_j+1) prefac
// (:660-662) times the colour filters' completeness (:666-668), shifted by the bias
// (:677-678) and binned in a left-closed histogram (:680, FP64 atomics); the nonzero bins
// become points at the bin centres with errors at the centres (:684-697) and are smoothed by
// the bin_cmd_smooth stamps (:702).  One thread per pair.
namespace {

constexpr int kPairThreads = 256;

// prefac[t] = norm[t] / mean_mass / 4 / trapz(m, imf(m)) (:642-643); one block per template,
// fixed-order block sum.
__global__ void __launch_bounds__(kPairThreads)
k_bin_prefac(IsoParams P, const double *__restrict__ m, const int64_t *__restrict__ off,
             const int32_t *__restrict__ len, const double *__restrict__ norm,
             double *__restrict__ prefac) {
    __shared__ double s_red[kPairThreads / 32];
    const int t = blockIdx.x, n = len[t];
    const double *mt = m + off[t];
    double acc = 0.0;
    for (int i = threadIdx.x; i + 1 < n; i += blockDim.x)
        acc += (mt[i + 1] - mt[i]) * (imf_pdf(P, mt[i]) + imf_pdf(P, mt[i + 1])) / 2.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int w = 0; w < kPairThreads / 32; ++w) tot += s_red[w];
        prefac[t] = norm[t] * P.inv_mean_mass / 4.0 / tot;
    }
}

// fluxes of the two colour filters, of which one is the magnitude filter (:644, :700), and
// IMF values.
__global__ void k_bin_flux(IsoParams P, const double *__restrict__ m, const double *__restrict__ mags,
                           int64_t total, double *__restrict__ fl, double *__restrict__ wv) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int fs[2] = {P.c1, P.c2};
#pragma unroll
    for (int q = 0; q < 2; ++q) fl[q * total + i] = exp10(-0.4 * mags[(int64_t)fs[q] * total + i]);
    // the interval's weight (of a template's last point: not used)
    if (i + 1 < total) wv[i] = (m[i + 1] - m[i]) * (imf_pdf(P, m[i]) + imf_pdf(P, m[i + 1]));
}

// left-closed histogram bin of v (edges first + k step, step > 0), -1 outside: the product with
// the inverse step, and the edges themselves only within 1e-6 bins of one
__device__ __forceinline__ int hist_bin(double v, double first, double step, double inv, int n) {
    const double q = (v - first) * inv;
    if (!(q >= -1.0 && q <= (double)n)) return -1;
    int k = __double2int_rd(q);
    const float frac = (float)(q - (double)k);
    if (frac < 1e-6f || frac > 1.f - 1e-6f) {
        if (!(v >= first)) return -1;
        k = max(k, 0);
        if (k > 0 && v < first + (double)k * step) --k;
        if (v >= first + (double)(k + 1) * step) ++k;
    }
    return (k >= 0 && k < n) ? k : -1;
}

// Natural logarithm by a table (Tang, 1990): x = 2^e c_j (1 + r), c_j = 1 + j / 128, and the
// series of log1p(r) to r^7 (|r| < 2^-7: the rest is below 2e-18).  About a dozen FP64
// operations; s_log[j] = (1 / c_j, log c_j).
__device__ __forceinline__ double log_table(double x, const double2 *s_log) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int e = (int)(b >> 52) - 1023, j = (int)(b >> 45) & 127;
    if (e < -1000 || e > 1000) return log(x);  // negative, subnormal, huge, inf or NaN
    const double m = __longlong_as_double((long long)((b & 0xfffffffffffffull) | 0x3ff0000000000000ull));
    const double c = __longlong_as_double((long long)((b & 0xfe00000000000ull) | 0x3ff0000000000000ull));
    const double2 t = s_log[j];
    const double r = (m - c) * t.x;
    double p = fma(r, 1.0 / 7.0, -1.0 / 6.0);
    p = fma(r, p, 1.0 / 5.0);
    p = fma(r, p, -1.0 / 4.0);
    p = fma(r, p, 1.0 / 3.0);
    p = fma(r, p, -1.0 / 2.0);
    return fma((double)e, 0.6931471805599453, t.y) + fma(r * r, p, r);
}

// -2.5 log10 x to 2e-9, as log2_fp32 (the same values out of range).
__device__ __forceinline__ double mag_fp32(double x, const double2 *s_log, const float2 *s_mag) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int e = (int)(b >> 52) - 1023, j = (int)(b >> 45) & 127;
    if (e < -1000 || e > 1000) return -1.0857362047581296 * log_table(x, s_log);
    const float c = __uint_as_float(0x3f800000u | (unsigned)j << 16);
    const float r = __fdividef((float)(unsigned)(b >> 13), c) * 1.8189894035458565e-12f;  // 2^-39
    const float2 t = s_mag[j];  // -2.5 log10 c_j as two floats
    const float l = fmaf(r * r, fmaf(r, fmaf(r, -0.25f, 1.f / 3.f), -0.5f), r);
    return fma((double)e, -0.7525749891599529, (double)t.x + (double)fmaf(l, -1.0857362f, t.y));
}

// hist_bin's axis, and how close to an edge a value known to 4e-9 can be binned with its position
// rounded to FP32: nearer than tol bins it may belong to either side.
struct BinAxis {
    double first, step, inv;
    int n;
    float tol;
    __device__ BinAxis(double f, double s, double i, int n_)
        : first(f), step(s), inv(i), n(n_), tol(1e-6f + 2.4e-7f * (float)n_ + 8e-9f * (float)fabs(i)) {}
    __device__ __forceinline__ int bin(double v, bool &near) const {
        const float q = (float)((v - first) * inv), k = floorf(q), out = fmaxf(1.f, tol);
        if (!(q > -out && q < (float)n + out)) return -1;
        near |= !(q - k > tol && q - k < 1.f - tol);
        return (q >= 0.f && q < (float)n) ? (int)k : -1;
    }
    __device__ __forceinline__ int exact(double v) const { return hist_bin(v, first, step, inv, n); }
};

// Grid: x -> left points i (a warp each), y -> template (chunk-relative); the lanes take the
// pairs' right points j.  hist is [chunk][nx*ny].  FP64 throughput bounds it: magnitudes take
// their logarithm's series in FP32, and the pairs nearer to a bin's edge than that and an FP32
// position can tell are binned from FP64 logarithms.  60 templates of 300 points: three library
// log10 and two divisions a pair 946 us, FP64 tables and positions 500 us, this way 255 us.
__global__ void __launch_bounds__(kPairThreads)
k_bin_pairs(IsoParams P, const double *__restrict__ fl, const double *__restrict__ wv, int64_t total,
            const int64_t *__restrict__ off, const int32_t *__restrict__ len,
            const double *__restrict__ prefac, Grid2 g, const sfh_df *__restrict__ tab, int t0,
            double *__restrict__ hist) {
    __shared__ double2 s_log[128];
    __shared__ float2 s_mag[128];
    if (threadIdx.x < 128) {
        const double lg = (double)tab[threadIdx.x].h + (double)tab[threadIdx.x].l;
        s_log[threadIdx.x] = make_double2(128.0 / (128.0 + (double)threadIdx.x), lg);
        const double mg = -1.0857362047581296 * lg;
        s_mag[threadIdx.x] = make_float2((float)mg, (float)(mg - (double)(float)mg));
    }
    __syncthreads();
    const int t = t0 + blockIdx.y, ns = len[t] - 1, lane = threadIdx.x & 31;
    const int64_t o = off[t];
    const double *wt = wv + o;
    const double *f1 = fl + o, *f2 = fl + total + o;
    double *h = hist + (int64_t)blockIdx.y * g.nx * g.ny;
    const double k = -1.0857362047581296, pre = prefac[t];  // flux2mag(f) = -2.5 log10 f (:656)
    const BinAxis ax(g.xf, g.xs, g.ixs, g.nx), ay(g.yf, g.ys, g.iys, g.ny);
    const double b1 = P.bias[P.c1], b2 = P.bias[P.c2], by = P.bias[P.y_index];
    const bool y1 = P.y_index == P.c1;  // the magnitude is one of the colour's (:700)
    const double cA = P.cA[P.c1] * P.cA[P.c2];
    for (int i = blockIdx.x * (kPairThreads / 32) + (threadIdx.x >> 5); i < ns;
         i += gridDim.x * (kPairThreads / 32)) {
        const double fi1 = f1[i], fi2 = f2[i], wi = wt[i] * pre;
        for (int j = i + 1 + lane; j < ns; j += 32) {
            const double s1 = fi1 + f1[j], s2 = fi2 + f2[j];
            const double m1 = mag_fp32(s1, s_log, s_mag), m2 = mag_fp32(s2, s_log, s_mag);
            bool near = false;
            int ix = ax.bin((m1 + b1) - (m2 + b2), near), iy = ay.bin((y1 ? m1 : m2) + by, near);
            if (near) {
                const double x1 = k * log_table(s1, s_log), x2 = k * log_table(s2, s_log);
                ix = ax.exact((x1 + b1) - (x2 + b2));
                iy = ay.exact((y1 ? x1 : x2) + by);
            }
            if (ix < 0 || iy < 0) continue;
            double w = wi * wt[j];
            // the product of the two colour filters' completeness (compl_eval) over one division
            const double e1 = (double)__expf((float)((m1 - P.cm50[P.c1]) * P.crho_inv[P.c1]));
            const double e2 = (double)__expf((float)((m2 - P.cm50[P.c2]) * P.crho_inv[P.c2]));
            w *= cA * rcp_nr((1.0 + e1) * (1.0 + e2));
            atomicAdd(h + ix + (int64_t)g.nx * iy, w);
        }
    }
}

// Nonzero bins of a segment of kSegBins bins: x -> segment, y -> template of the chunk.
constexpr int kSegBins = 4096;

__global__ void __launch_bounds__(kPairThreads)
k_bin_count(const double *__restrict__ hist, int64_t nbins, int32_t *__restrict__ cnt) {
    __shared__ int s_red[kPairThreads / 32];
    const double *h = hist + (int64_t)blockIdx.y * nbins;
    const int64_t k0 = (int64_t)blockIdx.x * kSegBins, k1 = min(nbins, k0 + kSegBins);
    int c = 0;
    for (int64_t k = k0 + threadIdx.x; k < k1; k += kPairThreads) c += h[k] != 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int tot = 0;
        for (int w = 0; w < kPairThreads / 32; ++w) tot += s_red[w];
        cnt[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = tot;
    }
}

// Records of the nonzero bins in bin order (x fastest): the segment's first point is number
// first[] of its template.  The bins are listed first, so that the FP64 work of a record is
// done by full warps (few bins of a segment hold pairs).
__global__ void __launch_bounds__(kPairThreads)
k_bin_points(IsoParams P, const double *__restrict__ hist, Grid2 g, const int64_t *__restrict__ start,
             const int32_t *__restrict__ first, int cov, StarRec *__restrict__ rec,
             StarKey *__restrict__ key, StarId *__restrict__ narrow, int *__restrict__ n_narrow) {
    __shared__ int s_list[kSegBins];
    __shared__ int s_red[kPairThreads / 32];
    const int64_t nbins = (int64_t)g.nx * g.ny;
    const double *h = hist + (int64_t)blockIdx.y * nbins;
    const int64_t k0 = (int64_t)blockIdx.x * kSegBins;
    const int len = (int)min(nbins - k0, (int64_t)kSegBins);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // a warp's share: consecutive bins, 32 at a time
    constexpr int kShare = kSegBins / (kPairThreads / 32);
    unsigned masks[kShare / 32];
    int mine = 0;
#pragma unroll
    for (int c = 0; c < kShare / 32; ++c) {
        const int k = warp * kShare + c * 32 + lane;
        masks[c] = __ballot_sync(0xffffffffu, k < len && h[k0 + k] != 0.0);
        mine += __popc(masks[c]);
    }
    if (lane == 0) s_red[warp] = mine;
    __syncthreads();
    int at = 0, all = 0;
#pragma unroll
    for (int v = 0; v < kPairThreads / 32; ++v) {
        at += v < warp ? s_red[v] : 0;
        all += s_red[v];
    }
#pragma unroll
    for (int c = 0; c < kShare / 32; ++c) {
        if (masks[c] >> lane & 1u) s_list[at + __popc(masks[c] & ((1u << lane) - 1u))] = warp * kShare + c * 32 + lane;
        at += __popc(masks[c]);
    }
    __syncthreads();
    const int q0 = first[(int64_t)blockIdx.y * gridDim.x + blockIdx.x];
    const int xc = (P.c1 != P.y_index) ? P.c1 : P.c2;
    for (int p = threadIdx.x; p < all; p += kPairThreads) {
        const int64_t k = k0 + s_list[p];
        const int ix = (int)(k % g.nx), iy = (int)(k / g.nx);
        // edges[k] + step / 2 (:688-689) with the edge correctly rounded by one fma and no
        // further contraction: the centre is a rounding tie of the stamp's pixel
        // (x - first) / step + 1 = k + 1.5, so its exact double decides the stamp's pixel
        const double cx = __dadd_rn(__fma_rn((double)ix, g.xs, g.xf), g.xs / 2.0);
        const double cy = __dadd_rn(__fma_rn((double)iy, g.ys, g.yf), g.ys / 2.0);
        const double xmag = (P.y_index == P.c1) ? cy - cx : cy + cx;  // :692-695
        StarRec r{};
        star_record(r, g, cx, cy, err_eval(P, xc, xmag), err_eval(P, P.y_index, cy), h[k], cov);
        {
            const int64_t s = start[blockIdx.y] + q0 + p;
            store_record(r, g, StarId{(int)blockIdx.y, q0 + p}, rec + s, key + s, narrow, n_narrow);
        }
    }
}

__global__ void k_mix_binary(const float *__restrict__ single, const float *__restrict__ binary,
                             const double *__restrict__ bmf, int64_t nbins, int64_t n,
                             float *__restrict__ out) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const double b = bmf[k / nbins];
    out[k] = (float)((double)single[k] * (1.0 - b) + b * (double)binary[k]);
}

}  // namespace

extern "C" int sfh_binary_hess_batch_dev(sfh_ctx *ctx, const double *d_m_ini, const double *d_mags,
                                         int64_t total_points, const int64_t *h_off,
                                         const int32_t *h_len, int64_t ntempl, int nf,
                                         int y_index, int c1, int c2, const sfh_err_model *err,
                                         const sfh_compl_model *compl_, const double *bias,
                                         const sfh_imf *imf, double mean_mass,
                                         const double *h_norm, double x_first, double x_step,
                                         int64_t nx, double y_first, double y_step, int64_t ny,
                                         float *d_models) {
    if (!ctx || !d_m_ini || !d_mags || !h_off || !h_len || !err || !compl_ || !imf || !h_norm ||
        !d_models || ntempl < 1 || ntempl > 65535 || total_points < 1 || nx < 1 || ny < 1)
        return SFH_ERR_ARG;
    if (!(x_step > 0) || !(y_step > 0))
        return sfh_set_error(ctx, SFH_ERR_ARG, "binary_hess: bin edges must increase");
    if (!(y_index == c1 || y_index == c2))  // :700
        return sfh_set_error(ctx, SFH_ERR_UNSUPPORTED,
                             "binary_hess for y_index not in color_indices is not implemented");
    IsoParams P;
    int rc = make_iso_params(ctx, nf, y_index, c1, c2, err, compl_, bias, imf, mean_mass,
                             total_points, P);
    if (rc) return rc;
    int nmax = 0;
    for (int64_t t = 0; t < ntempl; ++t) {
        if (h_len[t] < 3 || h_len[t] > 65536 || h_off[t] < 0 || h_off[t] + h_len[t] > total_points)
            return sfh_set_error(ctx, SFH_ERR_ARG, "binary_hess: isochrone lengths in [3, 65536]");
        nmax = h_len[t] > nmax ? h_len[t] : nmax;
    }
    SFH_CK(ctx, cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    const int64_t nbins = nx * ny;
    const int64_t chunk = std::max<int64_t>(1, std::min<int64_t>(ntempl, (256ll << 20) / (nbins * 8)));
    const int64_t nseg = (nbins + kSegBins - 1) / kSegBins;
    const int cov = y_index == c1 ? -1 : 1;  // :698
    // scratch: per-template inputs (one upload), fluxes, IMF values, prefactors, then the
    // chunk's starts, counts and firsts (one upload) and pair histograms; the records, whose
    // number is known after the count, go into the staging buffer
    std::vector<char> head;
    auto add = [&](const void *src, size_t bytes) {
        const size_t at = head.size();
        head.resize(at + sfh_align256(bytes), 0);
        if (src) std::memcpy(head.data() + at, src, bytes);
        return at;
    };
    const std::vector<int32_t> hcov((size_t)chunk, cov);
    const size_t o_norm = add(h_norm, ntempl * 8), o_off = add(h_off, ntempl * 8);
    const size_t o_len = add(h_len, ntempl * 4), o_cov = add(hcov.data(), chunk * 4);
    size_t at = head.size();
    auto carve = [&](size_t bytes) {
        const size_t o = at;
        at += sfh_align256(bytes);
        return o;
    };
    const size_t o_fl = carve(2 * total_points * 8), o_w = carve(total_points * 8), o_pre = carve(ntempl * 8);
    const size_t up = sfh_align256(256) + sfh_align256(chunk * 8) + sfh_align256(chunk * 4);
    const size_t o_up = carve(up + chunk * nseg * 4);  // narrow counter, starts, counts, firsts
    const size_t o_seg = carve(chunk * nseg * 4), o_hist = carve(chunk * nbins * 8);
    if ((rc = sfh_scratch_reserve(ctx, at))) return rc;
    char *b = (char *)ctx->scratch;
    const int64_t *d_off = (const int64_t *)(b + o_off);
    const int32_t *d_len = (const int32_t *)(b + o_len);
    double *fl = (double *)(b + o_fl), *wv = (double *)(b + o_w), *prefac = (double *)(b + o_pre);
    double *hist = (double *)(b + o_hist);
    SFH_CK(ctx, cudaMemcpyAsync(b, head.data(), head.size(), cudaMemcpyHostToDevice, st));
    k_bin_flux<<<(unsigned)((total_points + 255) / 256), 256, 0, st>>>(P, d_m_ini, d_mags, total_points,
                                                                    fl, wv);
    SFH_LAUNCHED(ctx);
    k_bin_prefac<<<(unsigned)ntempl, kPairThreads, 0, st>>>(P, d_m_ini, d_off, d_len,
                                                            (const double *)(b + o_norm), prefac);
    SFH_LAUNCHED(ctx);
    const Grid2 g = make_grid(x_first, x_step, nx, y_first, y_step, ny);
    std::vector<int32_t> seg((size_t)(chunk * nseg));
    std::vector<char> hup(up + (size_t)(chunk * nseg) * 4, 0);
    int64_t *starts = (int64_t *)(hup.data() + 256);
    int32_t *counts = (int32_t *)(hup.data() + 256 + sfh_align256(chunk * 8));
    int32_t *firsts = (int32_t *)(hup.data() + up);
    for (int64_t t0 = 0; t0 < ntempl; t0 += chunk) {
        const int64_t nc = std::min(chunk, ntempl - t0);
        SFH_CK(ctx, cudaMemsetAsync(hist, 0, nc * nbins * 8, st));
        const dim3 grid((unsigned)((nmax - 1 + kPairThreads / 32 - 1) / (kPairThreads / 32)), (unsigned)nc);
        k_bin_pairs<<<grid, kPairThreads, 0, st>>>(P, fl, wv, total_points, d_off, d_len,
                                                    prefac, g, ctx->d_df_tab, (int)t0, hist);
        SFH_LAUNCHED(ctx);
        k_bin_count<<<dim3((unsigned)nseg, (unsigned)nc), kPairThreads, 0, st>>>(hist, nbins,
                                                                                 (int32_t *)(b + o_seg));
        SFH_LAUNCHED(ctx);
        SFH_CK(ctx, cudaMemcpyAsync(seg.data(), b + o_seg, nc * nseg * 4, cudaMemcpyDeviceToHost, st));
        SFH_CK(ctx, cudaStreamSynchronize(st));
        int64_t tot = 0, maxcount = 0;
        for (int64_t q = 0; q < nc; ++q) {
            int32_t c = 0;
            for (int64_t k = 0; k < nseg; ++k) {
                firsts[q * nseg + k] = c;
                c += seg[(size_t)(q * nseg + k)];
            }
            starts[q] = tot;
            counts[q] = c;
            tot += c;
            maxcount = std::max<int64_t>(maxcount, c);
        }
        const size_t nodes = nx <= kMaxColumns && ny <= (1 << 20) ? node_bytes(g, nc) : 0;
        if ((rc = sfh_stage_reserve(ctx, StampWork::bytes(tot, nodes)))) return rc;
        SFH_CK(ctx, cudaMemcpyAsync(b + o_up, hup.data(), hup.size(), cudaMemcpyHostToDevice, st));
        StampWork work((char *)ctx->stage, tot, maxcount);
        work.made = true;
        work.n_narrow = (int *)(b + o_up);
        const int64_t *d_start = (const int64_t *)(b + o_up + 256);
        const int32_t *d_cnt = (const int32_t *)(b + o_up + 256 + sfh_align256(chunk * 8));
        k_bin_points<<<dim3((unsigned)nseg, (unsigned)nc), kPairThreads, 0, st>>>(
            P, hist, g, d_start, (const int32_t *)(b + o_up + up), cov, work.rec, work.key, work.narrow, work.n_narrow);
        SFH_LAUNCHED(ctx);
        rc = launch_stamps(ctx, StampStars{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, d_start,
                                           d_cnt, (const int32_t *)(b + o_cov)},
                           nc, g, nullptr, work, d_models + t0 * nbins);
        if (rc) return rc;
        SFH_CK(ctx, cudaStreamSynchronize(st));
    }
    return SFH_OK;
}

extern "C" int sfh_mix_binary_templates_dev(sfh_ctx *ctx, const float *d_single,
                                            const float *d_binary, const double *h_bmf,
                                            int64_t ntempl, int64_t nbins, float *d_out) {
    if (!ctx || !d_single || !d_binary || !h_bmf || !d_out || ntempl < 1 || nbins < 1)
        return SFH_ERR_ARG;
    SFH_CK(ctx, cudaSetDevice(ctx->device));
    double *d_bmf = nullptr;
    SFH_CK(ctx, cudaMalloc(&d_bmf, ntempl * 8));
    cudaMemcpyAsync(d_bmf, h_bmf, ntempl * 8, cudaMemcpyHostToDevice, ctx->stream);
    const int64_t n = ntempl * nbins;
    k_mix_binary<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(d_single, d_binary, d_bmf,
                                                                       nbins, n, d_out);
    ctx->launches++;
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    cudaFree(d_bmf);
    return e == cudaSuccess ? SFH_OK : sfh_cuda_error(ctx, e, "mix binary templates");
}
