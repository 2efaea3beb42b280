// fit.cu -- device BFGS driver for fit_templates (src/fitting/solvers.jl:172-221) and
// fit_templates_fast (:238-275).
//
// The reference minimises fg! with Optim.BFGS (inverse-Hessian BFGS, H0 = I, update skipped
// when sᵀy <= 0, alphaguess InitialStatic(1.0, scaled=true): the first trial step of each
// line search is min(1, |d|) / |d|, line search HagerZhang) over a transformed vector θ:
//   log MAP: r = exp(θ), f = fg!(r) - Σθ, g = G r - 1   (:180-187)
//   log MLE: r = exp(θ), f = fg!(r),      g = G r       (:188-194)
//   sqrt:    r = θ²,     f = fg!(r),      g = 2 θ G     (:257-263)
// Here the whole optimisation stays on the GPU.  One evaluation slot is five launches on the
// context stream:
//   k_fit_trial   (1 CTA)  new direction bookkeeping, θt = θ + α d, r = transform(θt)
//   fg!                    the single-vector kernel (one-pass for FP32 storage)
//   k_fit_eval    (1 CTA)  transformed f, g; line-search test; accept (s, y) or backtrack
//   k_fit_hgemv   (grid)   H y and H g, one warp per row, after an accepted step
//   k_fit_hupdate (grid)   rank-two BFGS update of H and the next direction d = -H g
// The host captures a few slots into a CUDA graph and replays it, reading the state back
// once per replay; a finished state turns the queued slots into no-ops (the fg! kernel
// reads the same flag).  The line search accepts a trial step on sufficient decrease (or
// Hager-Zhang's approximate Wolfe conditions) together with the curvature condition; a
// step that decreases f while the slope is still steep is kept and the step expanded
// (secant of φ', 2x to 10x), and a failed step backtracks (secant / quadratic
// interpolation) or falls back to the kept point.  It is not HagerZhang's bracketing, so
// the iterates differ from the reference's while the optimum they converge to does not.
#include <algorithm>
#include <cmath>

#include "sfh_internal.cuh"

namespace {

constexpr int kVecThreads = 1024;
constexpr int kRowWarps = 8;  // most rows of H per CTA of k_fit_hgemv / k_fit_hupdate
constexpr int kMaxBacktracks = 40;
constexpr int kMaxExpand = 10;
constexpr double kArmijo = 1e-4;
constexpr double kApproxEps = 1e-6, kSigma = 0.9, kDelta = 0.1;
// transform value of a general objective: it writes f(θt) to negLogL and ∇f(θt) to Graw
constexpr int kFitObjective = SFH_FIT_OBJECTIVE;

struct FitState {
    double f, f_prev, dg0, alpha, gnorm, xchange;
    double f_b, alpha_b;  // the last trial point that passed the decrease test while steep
    int64_t evals, iter;
    int backtracks, expansions, best_valid, status, done, first, accept, reset_h, newdir, skip;
};

struct FitVecs {
    double *theta, *g, *d, *theta_t, *r, *Graw, *s, *y, *Hy, *Hg, *negLogL, *theta_b, *g_b;
    double *H;  // nt x nt, symmetric
    int64_t nt;
    int transform;
    int max_iter;
    double g_abstol, f_reltol, x_abstol;
};

// Maximum of two values that are >= 0 or NaN, by their bits: a NaN is the largest.
__device__ __forceinline__ double nanmax(double a, double b) {
    return __longlong_as_double(max(__double_as_longlong(fabs(a)), __double_as_longlong(fabs(b))));
}

// What bounds the vector kernels is the serial chain of FP64: two operations retire per SM clock, a
// warp's instruction holds its scheduler's FP64 pipe for 64 clocks and eight warps take 128.  So
// sums of several values share their instructions, scalars are formed by one warp, comparisons of
// magnitudes use the bits, and each kernel's loads are issued together before its first branch.
// Microseconds within an evaluation of 240 templates, start to start of the next kernel, before /
// after: k_fit_eval with an accepted step 8.0 / 6.1, k_fit_hgemv 6.4 / 4.3, k_fit_hupdate 6.5 /
// 5.4, k_fit_trial with a new direction 5.1 / 3.8, each with 1.1 us between two kernels (as
// programmatic dependents of one another the whole fit took the same time).  A fit of 331
// evaluations: 11.6 ms / 10.2 ms.

// Tree sums of N = 2 or 4 values over a warp (pairs 16 lanes apart, then 8, 4, 2, 1): value k ends
// in lane 32 k / N.  While lanes still hold several values, half of them go on with one half of
// the values and the other half with the rest, so an instruction adds for all.
template <int N>
__device__ __forceinline__ double warp_sums(const double (&v)[N]) {
    static_assert(N == 2 || N == 4, "");
    const int l = threadIdx.x & 31;
    double u[N / 2];
    const bool up = (l & 16) != 0;
#pragma unroll
    for (int k = 0; k < N / 2; ++k) {
        const double send = up ? v[k] : v[k + N / 2], keep = up ? v[k + N / 2] : v[k];
        u[k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
    double t;
    if constexpr (N == 4) {
        const bool up8 = (l & 8) != 0;
        const double send = up8 ? u[0] : u[1], keep = up8 ? u[1] : u[0];
        t = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    } else {
        t = u[0] + __shfl_xor_sync(0xffffffffu, u[0], 8);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

// Sums of N values over the block: all threads call it, every lane of warp 0 gets the results (the
// others get nothing of use).  The order of a sum does not depend on the block's size while a
// thread holds one element.  sh: 32 N doubles, free again after the caller's next barrier.
template <int N>
__device__ __forceinline__ void block_sums(double (&v)[N], double *sh) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    double t = warp_sums<N>(v);
    if (l % (32 / N) == 0) sh[32 * (l / (32 / N)) + w] = t;
    __syncthreads();
    if (w == 0) {
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] = l < nw ? sh[32 * k + l] : 0.0;
        t = warp_sums<N>(v);
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] = __shfl_sync(0xffffffffu, t, 32 / N * k);
    }
}

// The same for NaN-propagating maxima of two magnitudes.
__device__ __forceinline__ void block_max(double (&v)[2], double *sh) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    const auto warp_max = [&]() {
        const bool up = l >= 16;
        double t = nanmax(up ? v[1] : v[0], __shfl_xor_sync(0xffffffffu, up ? v[0] : v[1], 16));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) t = nanmax(t, __shfl_xor_sync(0xffffffffu, t, o));
        return t;
    };
    double t = warp_max();
    if (l % 16 == 0) sh[2 * l + w] = t;
    __syncthreads();
    if (w == 0) {
        v[0] = l < nw ? sh[l] : 0.0;
        v[1] = l < nw ? sh[32 + l] : 0.0;
        t = warp_max();
        v[0] = __shfl_sync(0xffffffffu, t, 0);
        v[1] = __shfl_sync(0xffffffffu, t, 16);
    }
}

__device__ __forceinline__ double to_coeff(int transform, double th) {
    return transform == SFH_FIT_SQRT ? th * th : exp(th);
}

__global__ void k_fit_init(FitState *S, FitVecs V) {
    const int64_t nt = V.nt, total = nt * nt;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total;
         k += (int64_t)gridDim.x * blockDim.x)
        V.H[k] = (k / nt == k % nt) ? 1.0 : 0.0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *S = FitState{};
        S->status = -1;
        S->first = 1;
    }
}

__global__ void __launch_bounds__(kVecThreads) k_fit_trial(FitState *S, FitVecs V) {
    __shared__ double sh[64];
    __shared__ double s_alpha;
    __shared__ int s_descent;
    const int64_t nt = V.nt, i0 = threadIdx.x;
    // the thread's first element (the only one up to kVecThreads templates) and the state
    const bool own = i0 < nt;
    const double th0 = own ? V.theta[i0] : 0.0, g0 = own ? V.g[i0] : 0.0;
    double d0 = own ? V.d[i0] : 0.0;
    const int first = S->first, accept = S->accept, newdir = S->newdir;
    int reset = accept ? 0 : S->reset_h;  // an accepted step consumed the pending reset
    double alpha = S->alpha;
    if (S->done) {
        if (threadIdx.x == 0) S->skip = 1;
        return;
    }
    if (!first && newdir) {
        double sums[2] = {0.0, 0.0};
        if (own) {
            sums[0] += g0 * d0;
            sums[1] += d0 * d0;
        }
        for (int64_t i = i0 + blockDim.x; i < nt; i += blockDim.x) {
            sums[0] += V.g[i] * V.d[i];
            sums[1] += V.d[i] * V.d[i];
        }
        block_sums<2>(sums, sh);
        const auto step = [](double dd) {
            const double nd = sqrt(dd);
            return nd > 0.0 ? fmin(1.0, nd) / nd : 1.0;  // InitialStatic(1.0, scaled=true)
        };
        if (threadIdx.x < 32) {
            const double dg = sums[0], a = step(sums[1]);
            if (threadIdx.x == 0) {
                s_descent = dg < 0.0;
                s_alpha = a;
                S->dg0 = dg;
                S->backtracks = 0;
                S->expansions = 0;
                S->best_valid = 0;
            }
        }
        __syncthreads();
        if (!s_descent) {  // not a descent direction: steepest descent, H restarts at I
            double gg[2] = {0.0, 0.0};
            for (int64_t i = i0; i < nt; i += blockDim.x) {
                V.d[i] = -V.g[i];
                gg[0] += V.g[i] * V.g[i];
            }
            d0 = -g0;
            block_sums<2>(gg, sh);
            if (threadIdx.x < 32) {
                const double a = step(gg[0]);
                if (threadIdx.x == 0) {
                    s_alpha = a;
                    S->dg0 = -gg[0];
                }
            }
            __syncthreads();
            reset = 1;
        }
        alpha = s_alpha;
    }
    for (int64_t i = i0; i < nt; i += blockDim.x) {
        const double th = i == i0 ? th0 : V.theta[i];
        const double t = first ? th : th + alpha * (i == i0 ? d0 : V.d[i]);
        V.theta_t[i] = t;
        if (V.transform != kFitObjective)  // a general objective maps θ itself
            V.r[i] = to_coeff(V.transform, t);
    }
    if (threadIdx.x == 0) {
        S->alpha = alpha;
        S->newdir = 0;
        S->accept = 0;
        S->reset_h = reset;
        S->skip = 0;
        S->evals += 1;
    }
}

enum : int { kExpand, kBacktrack, kAccept, kAcceptBest };  // what an evaluation leads to

__global__ void __launch_bounds__(kVecThreads) k_fit_eval(FitState *S, FitVecs V) {
    __shared__ double sh[64], sh_max[64];
    __shared__ int s_next;
    const int64_t nt = V.nt, i0 = threadIdx.x;
    // the thread's first element (the only one up to kVecThreads templates) and the state
    const bool own = i0 < nt;
    const double th0 = own ? V.theta_t[i0] : 0.0, G0 = own ? V.Graw[i0] : 0.0, r0 = own ? V.r[i0] : 0.0,
                 d0 = own ? V.d[i0] : 0.0, g0 = own ? V.g[i0] : 0.0;
    const double negLogL = *V.negLogL;
    const int first = S->first, nexp = S->expansions, have_best = S->best_valid;
    const double f0 = S->f, alpha = S->alpha, dg0 = S->dg0, f_b = S->f_b, alpha_b = S->alpha_b;
    if (S->done) return;
    // transformed gradient at θt, in place of the raw one, and the slope φ'(α) = gtᵀd
    double sums[2] = {0.0, 0.0};  // Σθ, gtᵀd
    const auto gradient = [&](double th, double G, double r) {
        if (V.transform == kFitObjective) return G;  // the objective wrote the gradient of f in θ
        // (rounded products: not contracted into the differences they enter below)
        if (V.transform == SFH_FIT_SQRT) return __dmul_rn(G * 2.0, th);
        return V.transform == SFH_FIT_LOG_MAP ? G * r - 1.0 : __dmul_rn(G, r);
    };
    const bool logs = V.transform != kFitObjective && V.transform != SFH_FIT_SQRT;
    const double gt0 = gradient(th0, G0, r0);
    for (int64_t i = i0; i < nt; i += blockDim.x) {
        const bool here = i == i0;
        const double th = here ? th0 : V.theta_t[i];
        const double gt = here ? gt0 : gradient(th, V.Graw[i], V.r[i]);
        if (logs) sums[0] += th;
        V.Graw[i] = gt;
        if (!first) sums[1] += gt * (here ? d0 : V.d[i]);
    }
    block_sums<2>(sums, sh);
    double ft = 0.0;  // of use in warp 0
    if (threadIdx.x < 32) {
        const double sumth = sums[0], dgt = sums[1];
        ft = negLogL - (V.transform == SFH_FIT_LOG_MAP ? sumth : 0.0);
        int next = kAccept;
        if (!first) {
            const bool finite = fabs(ft) < INFINITY && fabs(dgt) < INFINITY;
            // sufficient decrease, or Hager-Zhang's approximate Wolfe conditions (slope reduced
            // to within [σ φ'(0), (2δ - 1) φ'(0)], σ = 0.9, δ = 0.1, and f at most ε |f| higher,
            // ε = 1e-6), which keep making progress where f differences fall below rounding
            const bool armijo = finite && ft <= f0 + kArmijo * alpha * dg0;
            const bool steep = dgt < kSigma * dg0;
            const bool approx = finite && ft <= f0 + kApproxEps * fabs(f0) && dgt >= kSigma * dg0 &&
                                dgt <= (2.0 * kDelta - 1.0) * dg0;
            const bool ok = armijo || approx;
            if (ok && steep && nexp < kMaxExpand) {
                // decrease but the slope is still steep (curvature condition fails): keep this
                // point and try further along d, as HagerZhang's bracketing expands
                next = kExpand;
                double a = dgt > dg0 ? alpha * dg0 / (dg0 - dgt) : 4.0 * alpha;  // secant of φ'
                a = fmin(fmax(a, 2.0 * alpha), 10.0 * alpha);
                if (threadIdx.x == 0) {
                    S->f_b = ft;
                    S->alpha_b = alpha;
                    S->best_valid = 1;
                    S->expansions = nexp + 1;
                    S->alpha = a;
                }
            } else if (!ok && have_best) {
                next = kAcceptBest;  // the expansion overshot: take the kept point
            } else if (!ok) {
                next = kBacktrack;
                if (threadIdx.x == 0) {
                    const int bt = S->backtracks + 1;
                    S->backtracks = bt;
                    double a = 0.5 * alpha;
                    if (finite) {
                        // root of the secant of φ' when the slope turned positive, else the
                        // minimiser of the quadratic through φ(0), φ'(0), φ(α)
                        const double q = dgt > 0.0
                                             ? alpha * dg0 / (dg0 - dgt)
                                             : -dg0 * alpha * alpha / (2.0 * (ft - f0 - dg0 * alpha));
                        a = fmin(fmax(q, 0.1 * alpha), 0.5 * alpha);
                        if (!(a == a)) a = 0.5 * alpha;
                    }
                    S->alpha = a;
                    if (bt >= kMaxBacktracks) {
                        S->status = SFH_FIT_LINESEARCH;
                        S->done = 1;
                    }
                }
            }
        }
        if (threadIdx.x == 0) s_next = next;
    }
    __syncthreads();
    const int next = s_next;
    if (next == kBacktrack) return;
    if (next == kExpand) {
        for (int64_t i = i0; i < nt; i += blockDim.x) {
            V.theta_b[i] = i == i0 ? th0 : V.theta_t[i];
            V.g_b[i] = i == i0 ? gt0 : V.Graw[i];
        }
        return;
    }
    const bool use_best = next == kAcceptBest;
    const double a_acc = use_best ? alpha_b : alpha;
    double most[2] = {0.0, 0.0};  // |g|, |s|
    for (int64_t i = i0; i < nt; i += blockDim.x) {
        const bool here = i == i0;
        const double gt = use_best ? V.g_b[i] : here ? gt0 : V.Graw[i];
        const double th = use_best ? V.theta_b[i] : here ? th0 : V.theta_t[i];
        if (first) {
            V.d[i] = -gt;
        } else {
            const double s = a_acc * (here ? d0 : V.d[i]);
            V.s[i] = s;
            V.y[i] = gt - (here ? g0 : V.g[i]);
            most[1] = nanmax(most[1], s);
        }
        V.theta[i] = th;
        V.g[i] = gt;
        most[0] = nanmax(most[0], gt);
    }
    const double f_acc = use_best ? f_b : ft;
    const bool flat = threadIdx.x < 32 && fabs(f0 - f_acc) <= V.f_reltol * fabs(f_acc);
    block_max(most, sh_max);
    const double gmax = most[0], smax = most[1];
    if (threadIdx.x == 0) {
        S->f_prev = first ? f_acc : f0;
        S->f = f_acc;
        S->gnorm = gmax;
        S->xchange = smax;
        S->newdir = 1;
        S->first = 0;
        int status = -1;
        if (!(fabs(f_acc) < INFINITY) || !(gmax < INFINITY)) {
            status = SFH_FIT_NONFINITE;
        } else if (gmax <= V.g_abstol) {
            status = SFH_FIT_CONVERGED_G;
        } else if (!first) {
            if (flat) status = SFH_FIT_CONVERGED_F;
            else if (smax <= V.x_abstol) status = SFH_FIT_CONVERGED_X;
        }
        if (!first) S->iter += 1;
        if (status < 0 && S->iter >= V.max_iter) status = SFH_FIT_MAXITER;
        // the inverse Hessian takes the accepted step even when it is the last one
        S->accept = (!first && status != SFH_FIT_NONFINITE) ? 1 : 0;
        if (status >= 0) {
            S->status = status;
            S->done = 1;
        }
    }
}

// Hy = H y, Hg = H g (H as I while a reset is pending), one warp per row.
__global__ void __launch_bounds__(kRowWarps * 32) k_fit_hgemv(const FitState *S, FitVecs V) {
    const int64_t nt = V.nt;
    const int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= nt) return;
    const int accept = S->accept, reset = S->reset_h;
    const double *row = V.H + i * nt;
    double a = 0.0, b = 0.0;
    for (int64_t j0 = 0; j0 < nt; j0 += 8 * 32) {  // eight columns' loads together
        double h[8], y[8], g[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int64_t j = j0 + 32 * u + lane;
            h[u] = j < nt ? row[j] : 0.0;
            y[u] = j < nt ? V.y[j] : 0.0;
            g[u] = j < nt ? V.g[j] : 0.0;
        }
        if (!accept) return;
        if (reset) break;
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (j0 + 32 * u + lane < nt) {
                a = fma(h[u], y[u], a);
                b = fma(h[u], g[u], b);
            }
    }
    if (reset) {
        if (lane == 0) {
            V.Hy[i] = V.y[i];
            V.Hg[i] = V.g[i];
        }
        return;
    }
    const double ab[2] = {a, b};
    const double t = warp_sums<2>(ab);
    if (lane == 0) V.Hy[i] = t;
    if (lane == 16) V.Hg[i] = t;
}

// H += c1 s sᵀ - c2 (Hy sᵀ + s Hyᵀ) with c1 = (sᵀy + yᵀHy) / (sᵀy)², c2 = 1 / sᵀy when
// sᵀy > 0 (Optim's BFGS update_h!), and d = -H_new g from the same vectors (contractions written
// out: the iterates' bits do not hang on the compiler's choice).  Every CTA
// forms the four dot products in the same order, so all see the same scalars.
// A CTA takes `rows` rows; its threads share their elements.
__global__ void __launch_bounds__(kRowWarps * 32) k_fit_hupdate(const FitState *S, FitVecs V, int rows) {
    __shared__ double sh[128];
    __shared__ double s_c[4];  // c1, c2, sᵀg, (Hy)ᵀg
    __shared__ int s_upd;
    const int64_t nt = V.nt, j0 = threadIdx.x;
    const bool own = j0 < nt;
    const double s0 = own ? V.s[j0] : 0.0, hy0 = own ? V.Hy[j0] : 0.0, g0 = own ? V.g[j0] : 0.0,
                 y0 = own ? V.y[j0] : 0.0;
    const int64_t i0 = (int64_t)blockIdx.x * rows;
    const int nr = (int)min((int64_t)rows, nt - i0);
    const int reset = S->reset_h;
    const double *vs = V.s, *vhy = V.Hy;
    const bool mine = (int)threadIdx.x < nr;
    const double my_hg = mine ? V.Hg[i0 + threadIdx.x] : 0.0, my_s = mine ? vs[i0 + threadIdx.x] : 0.0,
                 my_hy = mine ? vhy[i0 + threadIdx.x] : 0.0;
    if (!S->accept) return;
    double dots[4] = {0.0, 0.0, 0.0, 0.0};  // sᵀy, yᵀHy, sᵀg, (Hy)ᵀg
    for (int64_t j = j0; j < nt; j += blockDim.x) {
        const bool here = j == j0;
        const double s = here ? s0 : vs[j], hy = here ? hy0 : vhy[j], g = here ? g0 : V.g[j],
                     y = here ? y0 : V.y[j];
        dots[0] += s * y;
        dots[1] += y * hy;
        dots[2] += s * g;
        dots[3] += hy * g;
    }
    block_sums<4>(dots, sh);
    if (threadIdx.x < 32) {
        const double sty = dots[0], yhy = dots[1];
        const bool upd = sty > 0.0 && sty < INFINITY && fabs(yhy) < INFINITY;
        // c1 in lane 0 and c2 in the others by one division
        const bool l0 = threadIdx.x == 0;
        const double c = upd ? (l0 ? sty + yhy : 1.0) / (l0 ? sty * sty : sty) : 0.0;
        if (threadIdx.x < 2) s_c[threadIdx.x] = c;
        if (l0) {
            s_c[2] = dots[2];
            s_c[3] = dots[3];
            s_upd = upd;
        }
    }
    __syncthreads();
    const bool upd = s_upd != 0;
    const double c1 = s_c[0], c2 = s_c[1], sg = s_c[2], hyg = s_c[3];
    double *H = V.H + i0 * nt;
    if (upd || reset) {
        const int total = nr * (int)nt, step = kRowWarps * 32;  // rows <= 8, nt < 2^27
        for (int k0 = threadIdx.x; k0 < total; k0 += 4 * step) {
            double h[4], sj[4], hyj[4], si[4], hyi[4];  // four elements' loads before their stores
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = k0 + u * step;
                if (k >= total) break;
                const int r = k / (int)nt, j = k - r * (int)nt;
                h[u] = reset ? (j == i0 + r ? 1.0 : 0.0) : H[k];
                sj[u] = vs[j];
                hyj[u] = vhy[j];
                si[u] = vs[i0 + r];
                hyi[u] = vhy[i0 + r];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k0 + u * step < total)
                    H[k0 + u * step] = fma(-c2, fma(hyi[u], sj[u], __dmul_rn(si[u], hyj[u])),
                                           fma(__dmul_rn(c1, si[u]), sj[u], h[u]));
        }
    }
    if (mine)
        V.d[i0 + threadIdx.x] =
            -fma(-c2, fma(my_s, hyg, __dmul_rn(my_hy, sg)), fma(__dmul_rn(c1, my_s), sg, my_hg));
}

}  // namespace

// The BFGS loop over an objective: `objective` enqueues the evaluation at θt (nvar) on
// the context stream.  For the transforms of fit_templates it receives r = transform(θt)
// and writes fg!'s -logL and raw gradient; for kFitObjective it writes f(θt) and ∇f(θt).
// The slots are captured in a CUDA graph when the objective is capturable.
int sfh_bfgs_run(sfh_ctx *ctx, int64_t nvar, const double *d_theta0, const sfh_fit_options *opt,
                 int transform, const SfhFitObjective &objective, double *d_theta_out,
                 double *d_invH, sfh_fit_result *res) {
    if (opt->max_iter < 0 || !(opt->g_abstol >= 0.0) || !(opt->f_reltol >= 0.0) ||
        !(opt->x_abstol >= 0.0) || opt->max_evals < 0 || opt->graph_slots < 0 ||
        opt->graph_slots > 64 || !(opt->eps >= 0.0))
        return sfh_set_error(ctx, SFH_ERR_ARG, "invalid fit options");
    *res = sfh_fit_result{};
    const int64_t nt = nvar;
    const size_t vec = sfh_align256((size_t)nt * 8);
    const size_t o_state = 0, o_vecs = 256, o_H = o_vecs + 13 * vec, total = o_H + (size_t)nt * nt * 8;
    char *buf = nullptr;
    SFH_CK(ctx, cudaMalloc(&buf, total));
    FitState *S = (FitState *)(buf + o_state);
    double *v[13];
    for (int k = 0; k < 13; ++k) v[k] = (double *)(buf + o_vecs + k * vec);
    FitVecs V{v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10], v[11], v[12],
              (double *)(buf + o_H), nt, transform, opt->max_iter, opt->g_abstol,
              opt->f_reltol, opt->x_abstol};
    cudaStream_t st = ctx->stream;
    int rc = SFH_OK;
    const int64_t max_evals = opt->max_evals > 0 ? opt->max_evals : 50 * ((int64_t)opt->max_iter + 1);
    const int K = opt->graph_slots > 0 ? opt->graph_slots : 8;
    // rows per CTA: one CTA per SM (every CTA of k_fit_hupdate repeats four dot products), at
    // most eight rows
    const int rows = (int)std::max<int64_t>(1, std::min<int64_t>(kRowWarps, (nt + ctx->sm_count - 1) / ctx->sm_count));
    const int hgrid = (int)((nt + rows - 1) / rows);
    const int eval_threads = (int)std::min<int64_t>(kVecThreads, (nt + 31) / 32 * 32);
    auto slot = [&]() -> int {
        k_fit_trial<<<1, eval_threads, 0, st>>>(S, V);
        SFH_LAUNCHED(ctx);
        int r = objective(V.theta_t, V.r, V.Graw, V.negLogL, &S->skip);
        if (r) return r;
        k_fit_eval<<<1, eval_threads, 0, st>>>(S, V);
        SFH_LAUNCHED(ctx);
        k_fit_hgemv<<<hgrid, rows * 32, 0, st>>>(S, V);
        SFH_LAUNCHED(ctx);
        k_fit_hupdate<<<hgrid, kRowWarps * 32, 0, st>>>(S, V, rows);
        SFH_LAUNCHED(ctx);
        return SFH_OK;
    };
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    FitState h{};
    do {
        if ((rc = sfh_host_stage_reserve(ctx, sizeof(FitState)))) break;
        if (cudaMemcpyAsync(V.theta, d_theta0, nt * 8, cudaMemcpyDeviceToDevice, st) != cudaSuccess) {
            rc = sfh_cuda_error(ctx, cudaGetLastError(), "theta0 copy");
            break;
        }
        const int64_t ih = std::min<int64_t>((nt * nt + 255) / 256, 8 * (int64_t)ctx->sm_count);
        k_fit_init<<<(unsigned)std::max<int64_t>(ih, 1), 256, 0, st>>>(S, V);
        const cudaError_t e0 = cudaGetLastError();
        if (e0 != cudaSuccess) {
            rc = sfh_cuda_error(ctx, e0, "k_fit_init");
            break;
        }
        ctx->launches++;
        // the first evaluation runs eagerly (it also prepares the objective's plans and scratch)
        if ((rc = slot())) break;
        bool use_graph = true;
        int64_t per_replay = 0;  // kernels in one replay of the captured slots
        if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) use_graph = false;
        if (use_graph) {
            int r = SFH_OK;
            const int64_t l0 = ctx->launches;
            ctx->internal_capture = true;  // the graph lives only inside this call
            for (int k = 0; k < K && !r; ++k) r = slot();
            ctx->internal_capture = false;
            cudaError_t e = cudaStreamEndCapture(st, &graph);
            per_replay = ctx->launches - l0;
            ctx->launches = l0;  // captured, not launched: counted per replay below
            if (r || e != cudaSuccess || cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) {
                if (graph) cudaGraphDestroy(graph);
                graph = nullptr;
                exec = nullptr;
                cudaGetLastError();
                use_graph = false;
            }
        }
        res->graph = use_graph ? 1 : 0;
        for (;;) {
            if (cudaMemcpyAsync(ctx->h_stage, S, sizeof(FitState), cudaMemcpyDeviceToHost, st) !=
                    cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess) {
                rc = sfh_cuda_error(ctx, cudaGetLastError(), "fit state readback");
                break;
            }
            h = *(const FitState *)ctx->h_stage;
            if (h.done || h.evals >= max_evals) break;
            if (use_graph) {
                if (cudaGraphLaunch(exec, st) != cudaSuccess) {
                    rc = sfh_cuda_error(ctx, cudaGetLastError(), "fit graph launch");
                    break;
                }
                ctx->launches += per_replay;
            } else {
                for (int k = 0; k < K && !rc; ++k) rc = slot();
                if (rc) break;
            }
        }
        if (rc) break;
        if ((rc = sfh_check_onepass(ctx))) break;
        if (cudaMemcpyAsync(d_theta_out, V.theta, nt * 8, cudaMemcpyDeviceToDevice, st) != cudaSuccess ||
            (d_invH && cudaMemcpyAsync(d_invH, V.H, (size_t)nt * nt * 8, cudaMemcpyDeviceToDevice,
                                       st) != cudaSuccess) ||
            cudaStreamSynchronize(st) != cudaSuccess) {
            rc = sfh_cuda_error(ctx, cudaGetLastError(), "fit result copy");
            break;
        }
        res->f = h.f;
        res->g_norm = h.gnorm;
        res->iterations = h.iter;
        res->evaluations = h.evals;
        res->status = h.done ? h.status : SFH_FIT_MAXEVALS;
    } while (0);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    cudaStreamSynchronize(st);
    cudaFree(buf);
    return rc;
}

extern "C" int sfh_fit_bfgs_dev(sfh_ctx *ctx, sfh_models *m, const double *d_data,
                                const double *d_theta0, const sfh_fit_options *opt,
                                double *d_theta_out, double *d_invH, sfh_fit_result *res) {
    if (!ctx || !m || !d_data || !d_theta0 || !opt || !d_theta_out || !res) return SFH_ERR_ARG;
    if (opt->transform < SFH_FIT_LOG_MAP || opt->transform > SFH_FIT_SQRT)
        return sfh_set_error(ctx, SFH_ERR_ARG, "invalid fit options");
    SFH_CK(ctx, cudaSetDevice(ctx->device));
    double *comp = nullptr;
    SFH_CK(ctx, cudaMalloc(&comp, (size_t)m->nbins * 8));
    FgArgs a{};
    a.data = d_data;
    a.composite = comp;
    a.eps = opt->eps > 0.0 ? opt->eps : 2.220446049250313e-16;
    a.gsign = 1.0;
    a.mode = FG_MODE_FG;
    // fg! at r = transform(θt): -logL and the raw gradient G (k_fit_eval transforms them)
    SfhFitObjective fg = [&](const double *, double *r, double *Graw, double *negLogL,
                             const int *skip) -> int {
        FgArgs b = a;
        b.coeffs = r;
        b.G = Graw;
        b.negLogL = negLogL;
        b.skip = skip;
        return sfh_launch_fg(ctx, m, b);
    };
    const int rc = sfh_bfgs_run(ctx, m->nt, d_theta0, opt, opt->transform, fg, d_theta_out, d_invH, res);
    cudaStreamSynchronize(ctx->stream);
    cudaFree(comp);
    return rc;
}

// Host arrays: data (nbins), theta0 (nt) -> theta_out (nt), invH (nt x nt or NULL).
extern "C" int sfh_fit_bfgs(sfh_ctx *ctx, sfh_models *m, const double *data, const double *theta0,
                            const sfh_fit_options *opt, double *theta_out, double *invH,
                            sfh_fit_result *res) {
    if (!ctx || !m || !data || !theta0 || !opt || !theta_out || !res) return SFH_ERR_ARG;
    SFH_CK(ctx, cudaSetDevice(ctx->device));
    const int64_t nt = m->nt, nbins = m->nbins;
    const size_t o_th = sfh_align256((size_t)nbins * 8), o_out = o_th + sfh_align256((size_t)nt * 8),
                 o_H = o_out + sfh_align256((size_t)nt * 8),
                 total = o_H + (invH ? (size_t)nt * nt * 8 : 0);
    char *buf = nullptr;
    SFH_CK(ctx, cudaMalloc(&buf, total));
    cudaStream_t st = ctx->stream;
    int rc = SFH_OK;
    if (cudaMemcpyAsync(buf, data, nbins * 8, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(buf + o_th, theta0, nt * 8, cudaMemcpyHostToDevice, st) != cudaSuccess)
        rc = sfh_cuda_error(ctx, cudaGetLastError(), "fit input copy");
    if (!rc)
        rc = sfh_fit_bfgs_dev(ctx, m, (const double *)buf, (const double *)(buf + o_th), opt,
                              (double *)(buf + o_out), invH ? (double *)(buf + o_H) : nullptr, res);
    if (!rc && (cudaMemcpyAsync(theta_out, buf + o_out, nt * 8, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                (invH && cudaMemcpyAsync(invH, buf + o_H, (size_t)nt * nt * 8, cudaMemcpyDeviceToHost,
                                         st) != cudaSuccess) ||
                cudaStreamSynchronize(st) != cudaSuccess))
        rc = sfh_cuda_error(ctx, cudaGetLastError(), "fit output copy");
    cudaStreamSynchronize(st);
    cudaFree(buf);
    return rc;
}
