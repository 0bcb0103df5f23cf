// Preprocessing on the GPU: the sample moments of a daily-returns matrix and
// the realised crash frequency, in FP64.
//
// Replaces the reference's offline pandas steps:
//   compute_stats   preprocessing/preprocessing_stats.py:18,21
//                   mu = train.mean(), Sigma = train.cov() (ddof = 1)
//   compute_metrics preprocessing/evaluation.py:19,22
//                   fraction of days with (returns < -x).sum() >= k
//
// Moments, two passes like pandas' own covariance (means first, then the
// sum of products of deviations).  The bound is the FP64 pipe (64 cycles a
// warp instruction and sub-partition: about 256 multiply-adds a cycle over
// the chip), so the work, T N^2 / 2 multiply-adds (3.6e8 for 600 assets and
// 2000 days: 0.69 ms), is spread evenly and nothing else runs on that pipe:
//   col_sum    32 row segments x 32 columns a warp, Kahan-compensated; also
//              finds the first entry that is not finite (the host scan it
//              replaces took longer than the upload);
//   col_mean   a warp per column adds the 32 segments as (sum, error) pairs;
//   center     X - mu in place, once (centring the staged rows of every
//              tile cost 6 % of the covariance);
//   cov_tile   32 x 32 tiles of the lower triangle x row segments, enough
//              CTAs for about eight an SM (a CTA per tile left 38 of 152 SMs
//              with two tiles and the others with one);
//   cov_sum    segments added in order, scaled, mirrored.
// At T = 2000, N = 600 (under ncu): means 446 -> 37 us, covariance 1108 ->
// 655 + 8 + 12 us (centring, tiles, segment sums): the FP64 pipe's bound.
// Every output is summed in a fixed order, so results do not depend on
// scheduling.
#include <cmath>
#include <cstring>
#include "rg_internal.cuh"

namespace rg {

static constexpr int kMomTile = 32;
static constexpr int kMomSegs = 32; // row segments of the column sums
static constexpr unsigned long long kAllFinite = ~0ull;

__device__ __forceinline__ bool mom_finite(double v)
{
    return (__double_as_longlong(v) & 0x7ff0000000000000ll) != 0x7ff0000000000000ll;
}

// part[s][j], part[kMomSegs + s][j]: Kahan sum and correction of segment s of
// column j.  bad: smallest t n + j of an entry that is not finite.
__global__ void __launch_bounds__(256) col_sum_kernel(const double *__restrict__ X, long long T, int n,
                                                      double *__restrict__ part, unsigned long long *__restrict__ bad)
{
    const int j = blockIdx.x * 32 + (threadIdx.x & 31);
    const int seg = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (j >= n) return;
    const long long per = (T + kMomSegs - 1) / kMomSegs;
    const long long t0 = seg * per, t1 = min(T, t0 + per);
    double s = 0.0, c = 0.0;
    unsigned long long first = kAllFinite;
#pragma unroll 4
    for (long long t = t0; t < t1; t++) {
        const double x = X[t * n + j];
        if (!mom_finite(x)) first = min(first, (unsigned long long)(t * n + j));
        const double y = x - c;
        const double u = s + y;
        c = (u - s) - y;
        s = u;
    }
    part[(size_t)seg * n + j] = s;
    part[(size_t)(kMomSegs + seg) * n + j] = -c;
    if (first != kAllFinite) atomicMin(bad, first);
}

// One warp per column: lane = segment; the pairs (s, e) are added as a tree
// with the rounding error of every sum kept (Knuth's two-sum).
__global__ void __launch_bounds__(256) col_mean_kernel(const double *__restrict__ part, long long T, int n,
                                                       double *__restrict__ mu)
{
    const int j = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (j >= n) return;
    double s = part[(size_t)lane * n + j], e = part[(size_t)(kMomSegs + lane) * n + j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double b = __shfl_xor_sync(0xffffffffu, s, o), f = __shfl_xor_sync(0xffffffffu, e, o);
        const double u = s + b, v = u - s;
        e = (e + f) + ((s - (u - v)) + (b - v));
        s = u;
    }
    if (lane == 0) mu[j] = (s + e) / (double)T;
}

__global__ void center_kernel(double *__restrict__ X, long long T, int n, const double *__restrict__ mu)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const double m = mu[j];
    for (long long t = blockIdx.y; t < T; t += gridDim.y) X[t * n + j] -= m;
}

// Tile blockIdx.x of the lower triangle, rows [seg per, (seg + 1) per) of the
// centred matrix: part[seg][tile][32 x 32], or, with one segment, Sigma itself
// (the partials of many columns would be half of Sigma once more: N > 1536).
__global__ void __launch_bounds__(256) cov_tile_kernel(const double *__restrict__ X, long long T, int n,
                                                       long long per, double *__restrict__ part,
                                                       double *__restrict__ S)
{
    __shared__ double A[kMomTile][kMomTile + 1], B[kMomTile][kMomTile + 1];
    const int t = blockIdx.x;
    int bi = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((bi + 1) * (bi + 2) / 2 <= t) bi++;
    while (bi * (bi + 1) / 2 > t) bi--;
    const int bj = t - bi * (bi + 1) / 2;
    const int i0 = bi * kMomTile, j0 = bj * kMomTile;
    const int r = threadIdx.x >> 3, cb = (threadIdx.x & 7) * 4;
    const long long lo = blockIdx.y * per, hi = min(T, lo + per);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (long long t0 = lo; t0 < hi; t0 += kMomTile) {
        for (int e = threadIdx.x; e < kMomTile * kMomTile; e += blockDim.x) {
            const int tt = e / kMomTile, cc = e % kMomTile;
            const bool row_ok = t0 + tt < hi;
            A[tt][cc] = (row_ok && i0 + cc < n) ? X[(t0 + tt) * n + i0 + cc] : 0.0;
            B[tt][cc] = (row_ok && j0 + cc < n) ? X[(t0 + tt) * n + j0 + cc] : 0.0;
        }
        __syncthreads();
        const int rows = (int)min((long long)kMomTile, hi - t0);
#pragma unroll 4
        for (int tt = 0; tt < rows; tt++) {
            const double a = A[tt][r];
#pragma unroll
            for (int u = 0; u < 4; u++) acc[u] = fma(a, B[tt][cb + u], acc[u]);
        }
        __syncthreads();
    }
    if (gridDim.y == 1) {
        const double inv = 1.0 / (double)(T - 1);
#pragma unroll
        for (int u = 0; u < 4; u++) A[r][cb + u] = (0.0 + acc[u]) * inv; // as cov_sum_kernel adds one segment
        __syncthreads();
        for (int e = threadIdx.x; e < kMomTile * kMomTile; e += blockDim.x) {
            const int x = e / kMomTile, y = e % kMomTile;
            if (i0 + x < n && j0 + y < n) S[(long long)(i0 + x) * n + j0 + y] = A[x][y];
            if (bi != bj && i0 + y < n && j0 + x < n) S[(long long)(j0 + x) * n + i0 + y] = A[y][x];
        }
        return;
    }
    double *out = part + ((size_t)blockIdx.y * gridDim.x + t) * (kMomTile * kMomTile) + r * kMomTile + cb;
#pragma unroll
    for (int u = 0; u < 4; u++) out[u] = acc[u];
}

__global__ void __launch_bounds__(256) cov_sum_kernel(const double *__restrict__ part, int segs, long long T, int n,
                                                      double *__restrict__ S)
{
    __shared__ double tile[kMomTile][kMomTile + 1];
    const int t = blockIdx.x;
    int bi = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((bi + 1) * (bi + 2) / 2 <= t) bi++;
    while (bi * (bi + 1) / 2 > t) bi--;
    const int bj = t - bi * (bi + 1) / 2;
    const double inv = 1.0 / (double)(T - 1);
    for (int e = threadIdx.x; e < kMomTile * kMomTile; e += blockDim.x) {
        const int r = e / kMomTile, c = e % kMomTile, gi = bi * kMomTile + r, gj = bj * kMomTile + c;
        double v = 0.0;
        for (int s = 0; s < segs; s++) v += part[((size_t)s * gridDim.x + t) * (kMomTile * kMomTile) + e];
        v *= inv;
        tile[r][c] = v;
        if (gi < n && gj < n) S[(long long)gi * n + gj] = v;
    }
    if (bi == bj) return; // written in full above
    __syncthreads();
    for (int e = threadIdx.x; e < kMomTile * kMomTile; e += blockDim.x) {
        const int c = e / kMomTile, r = e % kMomTile, gi = bi * kMomTile + r, gj = bj * kMomTile + c;
        if (gi < n && gj < n) S[(long long)gj * n + gi] = tile[r][c];
    }
}

// One warp per day, lane = column: coalesced (a thread per day read rows
// apart: 64 us at T = 2000, N = 600, now 9).
__global__ void __launch_bounds__(256) crash_days_kernel(const double *__restrict__ X, long long T, int n,
                                                         double neg_x, int k, unsigned long long *__restrict__ days,
                                                         unsigned long long *__restrict__ bad)
{
    const long long t = blockIdx.x * 8ll + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= T) return;
    const double *row = X + t * n;
    int c = 0;
    unsigned long long first = kAllFinite;
    for (int j = lane; j < n; j += 32) {
        const double x = row[j];
        if (!mom_finite(x)) first = min(first, (unsigned long long)(t * n + j));
        c += (x < neg_x) ? 1 : 0;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0 && c >= k) atomicAdd(days, 1ull);
    if (first != kAllFinite) atomicMin(bad, first);
}

} // namespace rg

using namespace rg;

namespace {

int not_finite(int64_t t, int64_t j)
{
    return set_error(RG_ERR_INVALID, "returns[%lld][%d] is not finite", (long long)t, (int)j);
}

int check_matrix(const double *X, int64_t T, int32_t n, int64_t ld, int64_t min_rows)
{
    if (!X) return set_error(RG_ERR_INVALID, "returns is NULL");
    if (n < 1) return set_error(RG_ERR_INVALID, "n must be >= 1 (got %d)", n);
    if (T < min_rows) return set_error(RG_ERR_INVALID, "need at least %lld rows (got %lld)", (long long)min_rows, (long long)T);
    if (ld < n) return set_error(RG_ERR_INVALID, "ld (%lld) must be >= n (%d)", (long long)ld, n);
    return RG_OK;
}

// The kernels look for the first entry that is not finite.  Where they do not
// run (no device, no memory, a call that failed) the entries are checked here,
// so that bad input is reported as such before anything else.
int check_entries(const double *X, int64_t T, int32_t n, int64_t ld)
{
    for (int64_t t = 0; t < T; t++)
        for (int32_t j = 0; j < n; j++)
            if (!std::isfinite(X[t * ld + j])) return not_finite(t, j);
    return RG_OK;
}

int device_ready(const double *X, int64_t T, int32_t n, int64_t ld)
{
    int count = 0;
    if (cudaGetDeviceCount(&count) == cudaSuccess && count > 0) return RG_OK;
    cudaGetLastError();
    const int st = check_entries(X, T, n, ld);
    return st ? st : set_error(RG_ERR_NO_DEVICE, "no CUDA device is available");
}

// Rows packed to width n on the device.
cudaError_t upload(double *dX, const double *X, int64_t T, int32_t n, int64_t ld, cudaStream_t s)
{
    const size_t row = (size_t)n * sizeof(double);
    if (ld == n) return cudaMemcpyAsync(dX, X, row * (size_t)T, cudaMemcpyHostToDevice, s);
    return cudaMemcpy2DAsync(dX, row, X, (size_t)ld * sizeof(double), row, (size_t)T, cudaMemcpyHostToDevice, s);
}

} // namespace

extern "C" int rg_moments(const double *returns, int64_t T, int32_t n, int64_t ld, double *mu_out, double *sigma_out,
                          void *stream)
{
    int st = check_matrix(returns, T, n, ld, 2);
    if (st != RG_OK) return st;
    if (!mu_out || !sigma_out) return set_error(RG_ERR_INVALID, "mu_out / sigma_out is NULL");
    if ((st = device_ready(returns, T, n, ld)) != RG_OK) return st;
    cudaStream_t s = (cudaStream_t)stream;
    const int nb = (n + kMomTile - 1) / kMomTile, tiles = nb * (nb + 1) / 2;
    // about eight CTAs an SM, at least 64 rows each
    int64_t segs = (8 * kSms + tiles - 1) / tiles;
    if (segs > T / 64) segs = T / 64;
    if (segs > 64) segs = 64;
    if (segs < 1) segs = 1;
    const int64_t per = (T + segs - 1) / segs;
    segs = (T + per - 1) / per;
    // one allocation: X, mu, Sigma, column partials, tile partials, flag
    const size_t oX = 0, omu = oX + (size_t)T * n, oS = omu + (size_t)n, ocol = oS + (size_t)n * n,
                 ocov = ocol + 2 * (size_t)kMomSegs * n,
                 obad = ocov + (segs > 1 ? (size_t)segs * tiles * kMomTile * kMomTile : 0);
    double *d = nullptr;
    unsigned long long bad = kAllFinite;
    cudaError_t e = cudaSuccess;
    if ((st = pool_alloc((void **)&d, (obad + 1) * sizeof(double), s, &e)) != RG_OK)
        return check_entries(returns, T, n, ld) ? RG_ERR_INVALID : st;
    if (e == cudaSuccess) {
        unsigned long long *dbad = reinterpret_cast<unsigned long long *>(d + obad);
        e = cudaMemsetAsync(dbad, 0xff, sizeof(*dbad), s);
        if (e == cudaSuccess) e = upload(d + oX, returns, T, n, ld, s);
        if (e == cudaSuccess) {
            col_sum_kernel<<<dim3((n + 31) / 32, kMomSegs / 8), 256, 0, s>>>(d + oX, T, n, d + ocol, dbad);
            col_mean_kernel<<<(n + 7) / 8, 256, 0, s>>>(d + ocol, T, n, d + omu);
            const int gy = (int)(T < 256 ? T : 256);
            center_kernel<<<dim3((n + 127) / 128, gy), 128, 0, s>>>(d + oX, T, n, d + omu);
            cov_tile_kernel<<<dim3(tiles, (unsigned)segs), 256, 0, s>>>(d + oX, T, n, per, d + ocov, d + oS);
            if (segs > 1) cov_sum_kernel<<<tiles, 256, 0, s>>>(d + ocov, (int)segs, T, n, d + oS);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(&bad, dbad, sizeof(bad), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e == cudaSuccess && bad == kAllFinite) {
            e = cudaMemcpyAsync(mu_out, d + omu, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(sigma_out, d + oS, (size_t)n * n * sizeof(double), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        }
    }
    if (e != cudaSuccess) cudaStreamSynchronize(s); // no copy to or from the caller's memory stays in flight
    if (d) cudaFreeAsync(d, s);
    if (e != cudaSuccess && (st = check_entries(returns, T, n, ld)) != RG_OK) return st;
    if (e != cudaSuccess)
        return set_error(e == cudaErrorMemoryAllocation ? RG_ERR_NOMEM : RG_ERR_CUDA, "rg_moments: %s",
                         cudaGetErrorString(e));
    if (bad != kAllFinite) return not_finite((int64_t)(bad / (unsigned)n), (int64_t)(bad % (unsigned)n));
    return RG_OK;
}

extern "C" int rg_crash_frequency(const double *returns, int64_t T, int32_t n, int64_t ld, double x, int32_t k,
                                  double *freq_out, void *stream)
{
    int st = check_matrix(returns, T, n, ld, 1);
    if (st != RG_OK) return st;
    if (!freq_out) return set_error(RG_ERR_INVALID, "freq_out is NULL");
    if (!std::isfinite(x)) return set_error(RG_ERR_INVALID, "x must be finite");
    if ((st = device_ready(returns, T, n, ld)) != RG_OK) return st;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t xbytes = (size_t)T * (size_t)n * sizeof(double);
    unsigned char *d = nullptr;
    unsigned long long got[2] = {0, kAllFinite}; // crash days, first entry that is not finite
    cudaError_t e = cudaSuccess;
    if ((st = pool_alloc((void **)&d, xbytes + sizeof(got), s, &e)) != RG_OK)
        return check_entries(returns, T, n, ld) ? RG_ERR_INVALID : st;
    if (e == cudaSuccess) {
        unsigned long long *dgot = reinterpret_cast<unsigned long long *>(d + xbytes);
        e = cudaMemsetAsync(dgot, 0, sizeof(got[0]), s);
        if (e == cudaSuccess) e = cudaMemsetAsync(dgot + 1, 0xff, sizeof(got[1]), s);
        if (e == cudaSuccess) e = upload(reinterpret_cast<double *>(d), returns, T, n, ld, s);
        if (e == cudaSuccess) {
            crash_days_kernel<<<(unsigned)((T + 7) / 8), 256, 0, s>>>(reinterpret_cast<double *>(d), T, n, -x, k, dgot,
                                                                      dgot + 1);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(got, dgot, sizeof(got), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    if (e != cudaSuccess) cudaStreamSynchronize(s); // no copy to or from the caller's memory stays in flight
    if (d) cudaFreeAsync(d, s);
    if (e != cudaSuccess && (st = check_entries(returns, T, n, ld)) != RG_OK) return st;
    if (e != cudaSuccess)
        return set_error(e == cudaErrorMemoryAllocation ? RG_ERR_NOMEM : RG_ERR_CUDA, "rg_crash_frequency: %s",
                         cudaGetErrorString(e));
    if (got[1] != kAllFinite) return not_finite((int64_t)(got[1] / (unsigned)n), (int64_t)(got[1] % (unsigned)n));
    *freq_out = (double)got[0] / (double)T;
    return RG_OK;
}
