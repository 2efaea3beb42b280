// histogram.cu -- hard-binned Hess diagrams: bin_cmd (src/StarFormationHistories.jl:544-553),
// StatsBase's fit(Histogram, (colors, mags), Weights(w), edges; closed=:left).
//
// Bin k of an axis holds e[k] <= v < e[k+1] against the STORED edge values (StatsBase
// searches the range's own elements; a Julia range such as 0.0:0.1:1.0 holds 0.3 exactly,
// not 0 + 3 * 0.1).  A point on the last edge, below the first, or NaN is dropped.  A
// point's bin is guessed from the mean step and corrected against the edge values; blocks
// accumulate a private FP64 histogram in shared memory when the grid fits (dense photometric
// catalogues pile up in few bins) and flush it with global atomics.
#include <algorithm>
#include <cmath>

#include "sfh_internal.cuh"

namespace {

constexpr int kHistThreads = 256;
constexpr int64_t kHistSmemBins = 12288;  // 96 KB of FP64 bins per block

// FP64 arithmetic bounded the search (20 FP64 operations a point; the pipe retires two per SM
// clock): comparisons are made on the doubles' bits as integers, and the first guess in FP32.
// 2e6 points on 200 x 300 bins, data on the device: 92 us in FP64, 40 us this way.

// An integer that orders as the double does (-0 as +0; NaNs beyond the infinities).
__device__ __forceinline__ long long order_key(double v) {
    const long long b = __double_as_longlong(v);
    return b >= 0 ? b : (b == (long long)0x8000000000000000ull ? 0 : b ^ 0x7fffffffffffffffll);
}
// v as a float, by moving bits in the float's normal range (truncated: a guess only).
__device__ __forceinline__ float guess_float(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
    if (e < 897u || e > 1150u) return (float)v;
    return __uint_as_float(((unsigned)(b >> 32) & 0x80000000u) | ((e - 896u) << 23) |
                           (unsigned)((b >> 29) & 0x7fffffull));
}

struct HistAxis {
    const double *e;  // n + 1 increasing edges
    int n;
};

// One axis as a thread needs it: the first and last edges' keys and the mean inverse step.  far: the
// axis lies so far from zero that values in FP32 are several bins off (a time axis at 2.4e6 in steps of
// 1e-2); the difference to the first edge is then taken in FP64.  2e6 points, guesses from FP32 values /
// FP64 differences, us: 300 bins of 1 / 300 at 1e5 (3 bins off at most) 53 / 57, 300 bins of 0.01 at 2.45e6
// (24) 85 / 57, 4,000 bins of 5e-5 there (thousands) 6,190 / 57; near zero 50 / 57.
struct AxisGuess {
    long long first, last;
    double e0;
    float e0f, inv;
    bool far;
};
__device__ __forceinline__ AxisGuess axis_guess(const HistAxis &a) {
    const double e0 = a.e[0], e1 = a.e[a.n];
    const float e0f = (float)e0, inv = (float)((double)a.n / (e1 - e0));
    // (2^-22: a truncated value, the rounded edge and their difference; in FP32, since every thread
    // decides this)
    const float most = fmaxf(fabsf(e0f), fabsf((float)e1));
    return AxisGuess{order_key(e0), order_key(e1), e0, e0f, inv, !(most * 2.3841858e-7f * inv <= 8.f)};
}

// The bin of v, e[k] <= v < e[k + 1], or -1: the guess from the mean step, then a walk along
// the edges (a few steps at most on evenly spaced ones).  FAR: the guess from the FP64 difference.
template <bool FAR>
__device__ __forceinline__ int edge_bin(double v, const HistAxis &a, const AxisGuess &g) {
    const long long key = order_key(v);
    if (key < g.first || key >= g.last) return -1;
    const float d = FAR ? (float)(v - g.e0) : guess_float(v) - g.e0f;
    int k = (int)fminf(fmaxf(d * g.inv, 0.f), (float)(a.n - 1));
    k = min(k, a.n - 1);
    while (k > 0 && key < order_key(__ldg(a.e + k))) --k;
    while (k < a.n - 1 && key >= order_key(__ldg(a.e + k + 1))) ++k;
    return k;
}

struct HistAxes {
    HistAxis x, y;
};

// The thread's points, added to `to`.
template <bool FAR>
__device__ __forceinline__ void bin_points(const double *__restrict__ x, const double *__restrict__ y,
                                           const double *__restrict__ w, int64_t n, const HistAxes &A,
                                           const AxisGuess &gx, const AxisGuess &gy, double *to) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i0 < n; i0 += 4 * stride) {
        double vx[4], vy[4], vw[4];  // four points' loads in flight
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t i = i0 + u * stride;
            const bool have = i < n;
            vx[u] = have ? __ldcs(x + i) : __longlong_as_double(-1ll);  // a NaN: no bin
            vy[u] = have ? __ldcs(y + i) : 0.0;
            vw[u] = have && w ? __ldcs(w + i) : 1.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int ix = edge_bin<FAR>(vx[u], A.x, gx);
            if (ix < 0) continue;
            const int iy = edge_bin<FAR>(vy[u], A.y, gy);
            if (iy < 0) continue;
            atomicAdd(to + ix + (int64_t)A.x.n * iy, vw[u]);
        }
    }
}

// SHARED: a block's own FP64 histogram in shared memory, added to `out` at the end; else every
// point goes to `out` in L2.
template <bool SHARED>
__global__ void __launch_bounds__(kHistThreads, SHARED ? 4 : 6)
k_bin_cmd(const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ w,
          int64_t n, HistAxes A, double *__restrict__ out) {
    extern __shared__ double s_hist[];
    const AxisGuess gx = axis_guess(A.x), gy = axis_guess(A.y);
    double *to = SHARED ? s_hist : out;
    const int nb = A.x.n * A.y.n;
    if (SHARED) {
        for (int k = threadIdx.x; k < nb; k += blockDim.x) s_hist[k] = 0.0;
        __syncthreads();
    }
    // (two loops: a choice per point made every point pay for both guesses, 80 us instead of 50 for
    // 2e6 points)
    if (gx.far || gy.far) bin_points<true>(x, y, w, n, A, gx, gy, to);
    else bin_points<false>(x, y, w, n, A, gx, gy, to);
    if (SHARED) {
        __syncthreads();
        for (int k = threadIdx.x; k < nb; k += blockDim.x)
            if (s_hist[k] != 0.0) atomicAdd(out + k, s_hist[k]);
    }
}

int check_edges(sfh_ctx *ctx, const double *e, int64_t n) {
    for (int64_t k = 0; k <= n; ++k)
        if (!std::isfinite(e[k]) || (k > 0 && !(e[k] > e[k - 1])))
            return sfh_set_error(ctx, SFH_ERR_ARG, "bin edges must be finite and increasing");
    return SFH_OK;
}

}  // namespace

// Stream-ordered on ctx's stream; d_hist_out (nx * ny, column-major like the reference's
// Histogram weights) is overwritten.  Edges must be increasing (sfh_bin_cmd checks them;
// here the bin search stays inside the edge arrays whatever they hold).
extern "C" int sfh_bin_cmd_dev(sfh_ctx *ctx, const double *d_x, const double *d_y,
                               const double *d_w, int64_t n, const double *d_xedges, int64_t nx,
                               const double *d_yedges, int64_t ny, double *d_hist_out) {
    if (!ctx || !d_hist_out || !d_xedges || !d_yedges || n < 0 || nx < 1 || ny < 1 ||
        nx * ny > INT32_MAX || (n > 0 && (!d_x || !d_y)))
        return SFH_ERR_ARG;
    SFH_CK(ctx, cudaSetDevice(ctx->device));
    const int64_t nb = nx * ny;
    SFH_CK(ctx, cudaMemsetAsync(d_hist_out, 0, nb * 8, ctx->stream));
    if (n == 0) return SFH_OK;
    const HistAxes A{{d_xedges, (int)nx}, {d_yedges, (int)ny}};
    // four points a thread (their loads overlap), at most eight blocks per SM
    const int64_t want = (n + kHistThreads * 4 - 1) / (kHistThreads * 4);
    const bool shared = nb <= kHistSmemBins;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(want, (shared ? 4 : 8) * (int64_t)ctx->sm_count));
    const size_t smem = shared ? (size_t)nb * 8 : 0;
    if (smem > 48 * 1024)
        SFH_CK(ctx, cudaFuncSetAttribute(k_bin_cmd<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(kHistSmemBins * 8)));
    auto kern = shared ? k_bin_cmd<true> : k_bin_cmd<false>;
    kern<<<grid, kHistThreads, smem, ctx->stream>>>(d_x, d_y, d_w, n, A, d_hist_out);
    SFH_CK(ctx, cudaGetLastError());
    ctx->launches++;
    return SFH_OK;
}

// Host buffers: x, y, w (NULL = unit weights) of n points; xedges (nx + 1 values), yedges
// (ny + 1 values); hist_out (nx * ny).  Synchronous.
extern "C" int sfh_bin_cmd(sfh_ctx *ctx, const double *x, const double *y, const double *w,
                           int64_t n, const double *xedges, int64_t nx, const double *yedges,
                           int64_t ny, double *hist_out) {
    if (!ctx || !hist_out || !xedges || !yedges || n < 0 || nx < 1 || ny < 1 ||
        nx * ny > INT32_MAX || (n > 0 && (!x || !y)))
        return SFH_ERR_ARG;
    int rc = check_edges(ctx, xedges, nx);
    if (!rc) rc = check_edges(ctx, yedges, ny);
    if (rc) return rc;
    SFH_CK(ctx, cudaSetDevice(ctx->device));
    const int64_t nb = nx * ny;
    const size_t a = sfh_align256((size_t)(n > 0 ? n : 1) * 8);
    const size_t o_ex = 3 * a, o_ey = o_ex + sfh_align256((nx + 1) * 8),
                 o_out = o_ey + sfh_align256((ny + 1) * 8), total = o_out + nb * 8;
    rc = sfh_stage_reserve(ctx, total);
    if (rc) return rc;
    char *b = (char *)ctx->stage;
    if (n > 0) {
        SFH_CK(ctx, cudaMemcpyAsync(b, x, n * 8, cudaMemcpyHostToDevice, ctx->stream));
        SFH_CK(ctx, cudaMemcpyAsync(b + a, y, n * 8, cudaMemcpyHostToDevice, ctx->stream));
        if (w) SFH_CK(ctx, cudaMemcpyAsync(b + 2 * a, w, n * 8, cudaMemcpyHostToDevice, ctx->stream));
    }
    SFH_CK(ctx, cudaMemcpyAsync(b + o_ex, xedges, (nx + 1) * 8, cudaMemcpyHostToDevice, ctx->stream));
    SFH_CK(ctx, cudaMemcpyAsync(b + o_ey, yedges, (ny + 1) * 8, cudaMemcpyHostToDevice, ctx->stream));
    double *d_out = (double *)(b + o_out);
    rc = sfh_bin_cmd_dev(ctx, (const double *)b, (const double *)(b + a),
                         w ? (const double *)(b + 2 * a) : nullptr, n, (const double *)(b + o_ex),
                         nx, (const double *)(b + o_ey), ny, d_out);
    if (rc) return rc;
    SFH_CK(ctx, cudaMemcpyAsync(hist_out, d_out, nb * 8, cudaMemcpyDeviceToHost, ctx->stream));
    SFH_CK(ctx, cudaStreamSynchronize(ctx->stream));
    return SFH_OK;
}
