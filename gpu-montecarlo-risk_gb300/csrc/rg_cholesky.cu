// FP64 Cholesky factorisation of the covariance on the GPU.
//
// Replaces the host-side GSL factorisation of the reference wrapper
// (src/05-GPU/monte_carlos_cuda.cu:84-93, gsl_linalg_cholesky_decomp1) and
// its flatten step (:96-108, lower triangle kept, upper zeroed).  FP64 is
// kept for this one step: it is the step whose stability needs it.
//
// The FP64 pipe of this part takes 64 cycles for a warp instruction on one
// SM sub-partition (76 with all four busy), whether 32 lanes are active or
// one, so every form below spreads its FP64 warp instructions over warps and
// SMs and keeps the chain from one pivot to the next short.
//
// N <= 64 (chol_small_kernel): one CTA, right-looking, column by column: one
//   warp carries the chain from pivot to pivot, six apply the finished columns
//   to theirs (chol_factor_cta).
// Above (launch_cholesky_blocked): right-looking over 32-column blocks, two
//   launches a block:
//   chol_step   CTA 0 factors the next 32 x 32 diagonal block (the same
//               scheme); the other CTAs subtract the previous panel from the
//               rest of the trailing lower triangle, a 16 x 16 tile each, at
//               the same time;
//   chol_panel  one warp per row below the block solves x L_kk^T = a with a
//               lane per column: 32 steps of one shuffle and one FMA, on the
//               rows of L_kk divided by their pivots.  Its first cluster of
//               eight CTAs then subtracts its 32 rows' products from the next
//               diagonal block (in chol_step's CTA 0 they stood before the
//               pivots: N = 600 673 us instead of 552).
//   A 32 x 32 x 32 update is 19.5k cycles of one SM's FP64 pipe, hence the
//   16 x 16 tiles (N = 600: 663 in the first step), and a row per warp in the
//   panel (a row per lane put all 32 rows of a CTA on one sub-partition: 28 us
//   a panel at N = 600, now 9, both under ncu).  The launches overlap their
//   start-up with the previous kernel's end (programmatic dependent launch).
//   chol_prep (finite checks, lower(A), w32, per-row moment terms) runs
//   first, chol_finish (packed FP32 rows, moment sums in a fixed order, so
//   the result does not depend on scheduling) last.
// Device time of the factorisation, microseconds, before (the left-looking
// one-CTA form up to N = 64; above, one warp per diagonal block, a row per
// lane in the panel, 32 x 32 update tiles) and now:
//   N        9    20    50    64    65   200   333   600   1000   2000
//   before  34    65   178   249   188   538   924  1578   2810   7246
//   now     12    18    51    59    58   158   260   466    908   3289
// N = 64 is the widest block whose columns stay in registers.  The blocked form
// takes 16, 20, 44 and 50 us at N = 9, 20, 50 and 64, but subtracts the products
// one by one: its error there is larger than that of the form before (FINE).
// RG_CHOLESKY=single forces cholesky_kernel, one CTA left-looking column by
// column in place in the row-major output, above N = 64 too (a second
// implementation that the tests compare).
//
// A pivot that is not > 0 (or not finite) stops the factorisation and
// records info = column + 1 (every later kernel returns at once); the host
// turns that into RG_ERR_NOT_PD.  A non-finite input records info = -1
// (RG_ERR_INVALID).
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include "rg_internal.cuh"

namespace rg {

static constexpr int kCholThreads = 512;
static constexpr int kCholMaxN = 4096; // shared staging of one row: 32 KB

__device__ __forceinline__ double block_sum(double v, double *red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (warp == 0) {
        t = (lane < (int)(blockDim.x >> 5)) ? red[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

__global__ void __launch_bounds__(kCholThreads) cholesky_kernel(
    const double *__restrict__ A, long long lda, int n, const double *__restrict__ w,
    const double *__restrict__ mu, double *__restrict__ L, float *__restrict__ Lp,
    float *__restrict__ w32, double *__restrict__ aux, int *__restrict__ info)
{
    extern __shared__ double srow[]; // n doubles
    __shared__ double red[33];
    __shared__ double s_piv;
    __shared__ int s_fail;
    const int tid = threadIdx.x, bs = blockDim.x;

    // Every input that reaches the kernels must be finite (mu, weights, the
    // lower triangle of Sigma); info = -1 reports one that is not.
    int bad = 0;
    for (long long idx = tid; idx < (long long)n * n; idx += bs) {
        const int i = (int)(idx / n), j = (int)(idx % n);
        if (j <= i && !isfinite(A[(long long)i * lda + j])) bad = 1;
    }
    for (int i = tid; i < n; i += bs) {
        if (!isfinite(mu[i])) bad = 1;
        if (w != nullptr && !isfinite(w[i])) bad = 1;
        w32[i] = (w != nullptr) ? (float)w[i] : 0.f;
    }
    if (__syncthreads_or(bad)) {
        if (tid == 0) *info = -1;
        return;
    }

    // Portfolio moments from the input (lower triangle, symmetric use).
    if (w != nullptr) {
        double part = 0.0, pm = 0.0;
        for (long long idx = tid; idx < (long long)n * n; idx += bs) {
            const int i = (int)(idx / n), j = (int)(idx % n);
            const double a = (j <= i) ? A[(long long)i * lda + j] : A[(long long)j * lda + i];
            part += w[i] * a * w[j];
        }
        for (int i = tid; i < n; i += bs) pm += w[i] * mu[i];
        const double wsw = block_sum(part, red);
        const double wmu = block_sum(pm, red);
        if (tid == 0) { aux[0] = wsw; aux[1] = wmu; }
    } else if (tid == 0) {
        aux[0] = 0.0;
        aux[1] = 0.0;
    }

    // L <- lower(A), zero upper.
    for (long long idx = tid; idx < (long long)n * n; idx += bs) {
        const int i = (int)(idx / n), j = (int)(idx % n);
        L[idx] = (j <= i) ? A[(long long)i * lda + j] : 0.0;
    }
    if (tid == 0) s_fail = 0;
    __syncthreads();

    for (int j = 0; j < n; j++) {
        // stage row j (entries k < j are final) and form the pivot
        double part = 0.0;
        for (int k = tid; k < j; k += bs) {
            const double v = L[(long long)j * n + k];
            srow[k] = v;
            part += v * v;
        }
        const double ss = block_sum(part, red); // also orders srow writes before reads
        if (tid == 0) {
            const double d = L[(long long)j * n + j] - ss;
            if (!(d > 0.0) || !isfinite(d)) {
                s_fail = j + 1;
            } else {
                s_piv = sqrt(d);
                L[(long long)j * n + j] = s_piv;
            }
        }
        __syncthreads();
        if (s_fail) break;
        const double piv = s_piv;
        for (int i = j + 1 + tid; i < n; i += bs) {
            const double *row = L + (long long)i * n;
            double s0 = row[j], s1 = 0.0;
            int k = 0;
            for (; k + 1 < j; k += 2) {
                s0 = fma(-row[k], srow[k], s0);
                s1 = fma(-row[k + 1], srow[k + 1], s1);
            }
            if (k < j) s0 = fma(-row[k], srow[k], s0);
            L[(long long)i * n + j] = (s0 + s1) / piv;
        }
        __syncthreads();
    }
    if (tid == 0) *info = s_fail;
    if (s_fail) return;
    __syncthreads();

    // Packed FP32 rows (zero padded to multiples of 4).
    for (int i = tid; i < n; i += bs) {
        const int off = packed_row_offset(i), len = 4 * (i / 4 + 1);
        for (int j = 0; j < len; j++) Lp[off + j] = (j <= i) ? (float)L[(long long)i * n + j] : 0.f;
    }
}

static constexpr int kCholNb = 32;          // block size of the blocked form
static constexpr int kCholSmallMaxN = 64;   // the one-CTA form up to here
static constexpr int kCholCta = 256;        // threads of the factoring CTA and of chol_step's others
static constexpr int kCholTimeout = -2;     // info: a bounded wait ran out
static constexpr int kCholTile = 16;        // trailing-update tile
static constexpr size_t kCholAlone = 104 * 1024; // dynamic shared memory that, with the static, leaves one CTA an SM

// A positive finite pivot, tested on the bits (no FP64-pipe instruction).
__device__ __forceinline__ bool good_pivot(double d)
{
    const long long b = __double_as_longlong(d);
    return b > 0ll && b < 0x7ff0000000000000ll;
}
__device__ __forceinline__ bool finite_bits(double v)
{
    return (__double_as_longlong(v) & 0x7ff0000000000000ll) != 0x7ff0000000000000ll;
}

// 1 / sqrt(d) of a positive finite d, in integers: an FP64 instruction takes
// 64 cycles or more on the chain from pivot to pivot, where the Newton step in
// FP64 (five instructions) was the longest piece: 470 cycles a column of a
// 32-column block, now 340.  With d = x 2^(2k), 1 <= x < 4, y0 the hardware's
// FP32 approximation to 22 bits after the point and e = 1 - x y0^2 (|e| <
// 2^-20, exact to 2^-61), 1 / sqrt(x) = y0 (1 - e)^(-1/2) =
// y0 (1 + e/2 + 3/8 e^2) to 5/16 e^3 < 2^-61.
// Largest error over 2e7 arguments, on the CPU with the approximation off by
// up to 3 ulp: 0.507 ulp (the FP64 form: 0.996).
// `low`, where wanted: what the rounding to 53 bits left out, so that
// fma(v, result, v * low) is v / sqrt(d) rounded about once.
__device__ __forceinline__ double pivot_rsqrt(double d, double *low = nullptr)
{
    const uint64_t b = (uint64_t)__double_as_longlong(d);
    const int be = (int)(b >> 52); // biased exponent
    if (be < 64 || be > 1983) {
        const double rs = rsqrt(d), y = d * rs;
        if (low) *low = 0.5 * rs * fma(-fma(d, rs, -y), rs, fma(-y, rs, 1.0));
        return rs;
    }
    const int ex = be - 1023, odd = ex & 1, k = ex >> 1;
    float y0;
    asm("rsqrt.approx.ftz.f32 %0, %1;" // x cut to 24 bits
        : "=f"(y0)
        : "f"(__uint_as_float((uint32_t)(127 + odd) << 23 | ((uint32_t)(b >> 29) & 0x7fffffu))));
    const uint32_t y = __float_as_uint(y0 + 2.0f) & 0x7fffffu;                        // y0 2^22
    const uint64_t x = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << (10 + odd); // x 2^62
    const int64_t e = (int64_t)((1ull << 61) - __umul64hi(x, (uint64_t)y * y << 19));  // e 2^61
    const int es = (int)(e >> 12);                                                     // e 2^49
    const int64_t c = e + ((3 * (int)(((int64_t)es * es) >> 32)) >> 7);                // (e/2 + 3/8 e^2) 2^62
    const int64_t r = ((int64_t)y << 40) + (((int64_t)y * (c >> 2)) >> 20);            // 2^62 / sqrt(x)
    // 53 bits, rounded; a carry out of them raises the exponent
    const uint64_t h = (uint64_t)(r + 256) >> 9;
    if (low) {
        const int l = (int)(r - (int64_t)(h << 9)); // times 2^(-62 - k)
        const uint64_t lb = (uint64_t)__double_as_longlong((double)l);
        *low = __longlong_as_double(l ? (long long)(lb - ((uint64_t)(62 + k) << 52)) : 0ll);
    }
    return __longlong_as_double((long long)(((uint64_t)(1021 - k) << 52) + h));
}

// The warps that factor a block: the chain warp (0) and six bulk warps (1-3,
// 5-7).  Warp 4 would share the chain warp's SM sub-partition, and its FP64
// instructions would queue ahead of the chain's: it does not take part.
static constexpr int kCholBulk = 6;
__device__ __forceinline__ bool chol_takes_part() { return (threadIdx.x >> 5) != 4; }

// Hand-over of columns between the warps of the factoring CTA: one mbarrier
// a column and direction, each used once.
struct CholFlags {
    unsigned long long fin[64]; // column final (chain -> bulk)
    unsigned long long pre[64]; // column up to date but for the two before it (bulk -> chain)
};
__device__ __forceinline__ unsigned chol_smem(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void chol_flags_init(CholFlags &f)
{
    for (int i = threadIdx.x; i < 64; i += blockDim.x) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(chol_smem(&f.fin[i])) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(chol_smem(&f.pre[i])) : "memory");
    }
}
// The whole warp's writes before it are visible to the waiters.
__device__ __forceinline__ void chol_arrive(unsigned long long *bar)
{
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(chol_smem(bar)) : "memory");
}
// Bounded: false after about a second (the other warps of the CTA are
// resident, so a wait ends within microseconds unless something is broken).
__device__ __forceinline__ bool chol_wait(unsigned long long *bar)
{
    for (int i = 0; i < (1 << 20); i++) {
        unsigned ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(chol_smem(bar))
                     : "memory");
        if (ok) return true;
    }
    return false;
}

// Factor an n x n block (n <= NC) in place: col[c NR + row], NR = NC rounded
// up to 32, lower triangle, zeros above the diagonal; the reciprocal pivots
// are left in inv[].  Called by the seven warps of a 256-thread CTA that take
// part, after a barrier that made col and the initialised flags visible and
// *s_fail zero; another CTA barrier must follow.  *s_fail is then 0, 1 + the
// first failing column, or -1 (a bounded wait ran out).
//
// Right-looking.  The chain warp, once column c - 1 is final and column c has
// had every column before c - 2 applied, applies columns c - 2 and c - 1, forms
// the pivot and leaves column c final: two FMAs, the reciprocal square root and
// one multiply (FINE: and an FMA) a column.  (With column c - 2 left to the bulk warps too, the
// chain waited for them 280 of 1220 cycles a column of a 32-column block
// instead of 140 of 930.)  The bulk warps
// (column j in the registers of bulk warp j mod 6, lane = row, two rows a lane
// for NC > 32) apply each final column c to theirs; the one that owns column
// c + 3 does that one first, writes it
// back for the chain warp and catches up with its other columns later
// (`done`: columns applied so far).  Hand-over by column instead of a CTA
// barrier a column lets a bulk warp fall behind while the chain goes on.
//
// FINE (N <= 64) keeps the error of the form before, the left-looking one with
// sums of their own, a square root and divisions: the quotients are rounded
// about once (pivot_rsqrt's low part), and the bulk warps sum a column's products
// from zero in four parts and subtract them from it once.
// Root-mean-square error of L against extended precision, in 2^-52 of L, over 12
// factor covariances a size (the form before; with products subtracted one by
// one and rounded reciprocals; now): N = 9 0.28, 0.37, 0.28; N = 20 0.41, 0.53,
// 0.43; N = 50 0.90, 0.91, 0.70; N = 64 1.12, 1.07, 0.92.  Device time, without
// FINE and with it, us: 10.4 and 11.7, 18.0 and 17.9, 47.1 and 50.6, 56.8 and
// 58.9.  Above 64 the two forms' errors are alike (N = 100 2.02 and 2.07, N = 200
// 3.68 and 3.67).
template <int NC, bool FINE>
__device__ __forceinline__ void chol_factor_cta(int n, double *col, double *inv, CholFlags &f, int *s_fail)
{
    constexpr int STEP = 2;
    constexpr int SL = (NC + kCholBulk - 1) / kCholBulk, G = (NC + 31) / 32, NR = 32 * G;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int *failed = s_fail;
    if (warp == 0) {
        double p[G], q[G]; // the previous column and the one before it
#pragma unroll
        for (int g = 0; g < G; g++) p[g] = q[g] = 0.0;
        // column c in the 32-row groups from `first` on (rows above the column's
        // own group hold nothing); false: given up
        auto column = [&](int c, auto first) -> bool {
            constexpr int g0 = decltype(first)::value;
            const double lp = -__shfl_sync(0xffffffffu, c >= 32 ? p[G - 1] : p[0], c & 31);
            const double lq = -__shfl_sync(0xffffffffu, c >= 32 ? q[G - 1] : q[0], c & 31);
            if (c >= 3 && !chol_wait(&f.pre[c])) {
                if (lane == 0) *failed = -1;
                return false;
            }
            double v[G];
#pragma unroll
            for (int g = g0; g < G; g++) {
                v[g] = fma(p[g], lp, fma(q[g], lq, col[c * NR + 32 * g + lane]));
                q[g] = p[g];
            }
            const double d = __shfl_sync(0xffffffffu, v[g0], c & 31);
            if (!good_pivot(d)) { // the same value in every lane
                if (lane == 0) *failed = c + 1;
                return false;
            }
            double low = 0.0;
            const double rs = pivot_rsqrt(d, FINE ? &low : nullptr);
#pragma unroll
            for (int g = g0; g < G; g++) {
                const double x = FINE ? fma(v[g], rs, v[g] * low) : v[g] * rs;
                p[g] = 32 * g + lane >= c ? x : 0.0; // on the diagonal d / sqrt(d)
                col[c * NR + 32 * g + lane] = p[g];
            }
            if (lane == 0) inv[c] = rs;
            chol_arrive(&f.fin[c]);
            return true;
        };
        int c = 0;
        bool ok = true;
        for (; ok && c < n && c < 32; c += ok) ok = column(c, std::integral_constant<int, 0>());
        for (; ok && c < n; c += ok) ok = column(c, std::integral_constant<int, G - 1>());
        // after a failure: release the bulk warps from the columns not
        // published (each flag is arrived on once)
        for (; c < n; c++) chol_arrive(&f.fin[c]);
        return;
    }
    const int b = warp < 4 ? warp - 1 : warp - 2; // bulk index
    // FINE: four sums of the columns' products, column k's in sum k mod 4;
    // else one, the column so far.  (Arrays of their own: chosen from by an
    // index known only at run time, one array would move to local memory.)
    double a[SL][G], a1[SL][G], a2[SL][G], a3[SL][G];
#pragma unroll
    for (int s = 0; s < SL; s++)
#pragma unroll
        for (int g = 0; g < G; g++) {
            const int j = s * kCholBulk + b;
            a[s][g] = !FINE && j < n ? col[j * NR + 32 * g + lane] : 0.0;
            a1[s][g] = a2[s][g] = a3[s][g] = 0.0;
        }
    // acc += (FINE) or -= column k's products, for the slots from s0 on
    auto apply = [&](int k, int s0, double (&acc)[SL][G]) {
        const double *ck = col + k * NR;
        double lr[G];
#pragma unroll
        for (int g = 0; g < G; g++) lr[g] = ck[32 * g + lane];
#pragma unroll
        for (int s = 0; s < SL; s++) {
            if (s < s0) continue;
            const int j = s * kCholBulk + b;
            const double l = FINE ? ck[j < NR ? j : 0] : -ck[j < NR ? j : 0];
            // rows above the column's own 32-row group hold nothing
#pragma unroll
            for (int g = 0; g < G; g++)
                if (g >= s * kCholBulk / 32) acc[s][g] = fma(lr[g], l, acc[s][g]);
        }
    };
    int done = 0;
    // Unrolled over the slots, two a step, so that finished columns cost little:
    // an FP64 instruction whose predicate is false still takes its 64 cycles.
    // One slot a step is more code to fetch (N = 600 478 us instead of 472), three
    // cost more finished columns (N = 50 52.7 instead of 50.7).
#pragma unroll
    for (int s0 = 0; s0 < SL; s0 += STEP) {
        for (int c = s0 * kCholBulk; c < (s0 + STEP) * kCholBulk && c + 3 < n; c++) {
            if (!chol_wait(&f.fin[c])) {
                if (lane == 0) *failed = -1;
                return;
            }
            if (*failed != 0) return;
            if (b == (c + 3) % kCholBulk) {
                // the owned column by masks, as above; its groups from g0 on
                const int g0 = (s0 * kCholBulk + 3) / 32;
                auto owned = [&](const double (&acc)[SL][G], double (&v)[G]) {
#pragma unroll
                    for (int g = g0; g < G; g++) {
                        long long bits = 0;
#pragma unroll
                        for (int s = s0; s < SL && s <= s0 + STEP; s++)
                            bits |= __double_as_longlong(acc[s][g]) & -(long long)(s == (c + 3) / kCholBulk);
                        v[g] = __longlong_as_double(bits);
                    }
                };
                double v[G], v1[G], v2[G], v3[G];
                owned(a, v);
                if (FINE) {
                    owned(a1, v1);
                    owned(a2, v2);
                    owned(a3, v3);
                }
                // (the columns before c have been applied: a warp's own columns
                // are kCholBulk apart; as a loop over the columns left to do
                // this one step took N = 600 from 472 to 544 us)
                const double l = FINE ? col[c * NR + c + 3] : -col[c * NR + c + 3];
#pragma unroll
                for (int g = g0; g < G; g++) v[g] = fma(col[c * NR + 32 * g + lane], l, v[g]);
#pragma unroll
                for (int g = g0; g < G; g++) {
                    double *x = col + (c + 3) * NR + 32 * g + lane;
                    *x = FINE ? *x - ((v[g] + v1[g]) + (v2[g] + v3[g])) : v[g];
                }
                chol_arrive(&f.pre[c + 3]);
                continue;
            }
            for (int k = done; k <= c; k++) {
                if (!FINE || (k & 3) == 0) apply(k, s0, a);
                else if ((k & 3) == 1) apply(k, s0, a1);
                else if ((k & 3) == 2) apply(k, s0, a2);
                else apply(k, s0, a3);
            }
            done = c + 1;
        }
    }
}

// N <= 64: everything in one CTA (NC = 16, 32, 48 or 64).
template <int NC>
__global__ void __launch_bounds__(kCholCta, 1) chol_small_kernel(
    const double *__restrict__ A, long long lda, int n, const double *__restrict__ w,
    const double *__restrict__ mu, double *__restrict__ L, float *__restrict__ Lp,
    float *__restrict__ w32, double *__restrict__ aux, int *__restrict__ info)
{
    constexpr int G = (NC + 31) / 32, NR = 32 * G, kW = kCholCta / 32, SEG = kW / G;
    __shared__ double col[NC * NR];
    __shared__ double sw[NR], smu[NR], inv[NC], part[SEG][NR];
    __shared__ CholFlags flags;
    __shared__ int s_fail;
    const int tid = threadIdx.x, bs = blockDim.x, warp = tid >> 5, lane = tid & 31;

    int bad = 0;
    for (int idx = tid; idx < NR * NC; idx += bs) {
        const int i = idx / NC, j = idx % NC;
        const double v = (i < n && j <= i) ? A[(long long)i * lda + j] : 0.0;
        if (!finite_bits(v)) bad = 1;
        col[j * NR + i] = v;
    }
    chol_flags_init(flags);
    if (tid == 0) s_fail = 0;
    for (int i = tid; i < NR; i += bs) {
        const double wi = (w != nullptr && i < n) ? w[i] : 0.0, mi = i < n ? mu[i] : 0.0;
        if (!finite_bits(wi) || !finite_bits(mi)) bad = 1;
        sw[i] = wi;
        smu[i] = mi;
        if (i < n) w32[i] = (float)wi;
    }
    if (__syncthreads_or(bad)) {
        if (tid == 0) *info = -1;
        return;
    }
    if (chol_takes_part()) chol_factor_cta<NC, true>(n, col, inv, flags, &s_fail);
    __syncthreads();
    if (tid == 0) *info = s_fail < 0 ? kCholTimeout : s_fail;
    if (s_fail) return;

    // L (zero upper) and the packed FP32 rows
    for (int idx = tid; idx < n * n; idx += bs) {
        const int i = idx / n, j = idx % n;
        L[idx] = j <= i ? col[j * NR + i] : 0.0;
    }
    for (int i = warp; i < n; i += kW) {
        const int off = packed_row_offset(i), len = 4 * (i / 4 + 1);
        for (int j = lane; j < len; j += 32) Lp[off + j] = j <= i ? (float)col[j * NR + i] : 0.f;
    }
    // w^T Sigma w (the strict lower triangle counts twice) and w.mu: lane =
    // row, a segment of its columns per warp
    if (w != nullptr) {
        constexpr int W = NR / SEG;
        const int i = 32 * (warp % G) + lane, seg = warp / G;
        double t = 0.0;
        for (int j = seg * W; j < (seg + 1) * W && j < n; j++)
            t = fma((i < n && j < i) ? A[(long long)i * lda + j] : 0.0, sw[j], t);
        part[seg][i] = 2.0 * t;
        __syncthreads();
        if (warp == 0) {
            double x = 0.0, y = 0.0;
#pragma unroll
            for (int g = 0; g < G; g++) {
                const int r = 32 * g + lane;
                double u = r < n ? A[(long long)r * lda + r] * sw[r] : 0.0;
#pragma unroll
                for (int q = 0; q < SEG; q++) u += part[q][r];
                x = fma(sw[r], u, x);
                y = fma(sw[r], smu[r], y);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                x += __shfl_xor_sync(0xffffffffu, x, o);
                y += __shfl_xor_sync(0xffffffffu, y, o);
            }
            if (lane == 0) {
                aux[0] = x;
                aux[1] = y;
            }
        }
    } else if (tid == 0) {
        aux[0] = 0.0;
        aux[1] = 0.0;
    }
}

// ------------------------------------------------------------ blocked form
// Start of a kernel launched programmatically behind the previous one: let
// the next one be scheduled, then wait until the previous one's writes are
// visible.  Such a kernel runs while its predecessor still writes L, dinv and
// info, so none of its pointers is __restrict__: that (with const, the
// read-only cache too) would let a load be placed before the wait.
__device__ __forceinline__ void pdl_enter()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Checks, L <- lower(A) (upper zeroed), w32, and the per-row moment terms
// aux[2 + i] = w_i (2 sum_{j<i} Sigma_ij w_j + Sigma_ii w_i),
// aux[2 + n + i] = w_i mu_i.  One warp per row (only the lower triangle is
// read: coalesced).
__global__ void chol_prep_kernel(const double *__restrict__ A, long long lda, int n, const double *__restrict__ w,
                                 const double *__restrict__ mu, double *__restrict__ L, float *__restrict__ w32,
                                 double *__restrict__ aux, int *__restrict__ info)
{
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    int bad = 0;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
        const double *ai = A + (long long)i * lda;
        double part = 0.0;
        for (int j0 = 0; j0 < n; j0 += 32) {
            const int j = j0 + lane;
            const double a = j <= i ? ai[j] : 0.0;
            if (!finite_bits(a)) bad = 1;
            if (j < n) L[(long long)i * n + j] = a;
            if (w != nullptr && j0 <= i) part = fma(a, j < i ? w[j] : 0.0, part);
        }
        double wi = 0.0, mi = 0.0;
        if (w != nullptr) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
            wi = w[i];
        }
        mi = mu[i];
        if (!finite_bits(wi) || !finite_bits(mi)) bad = 1;
        if (lane == 0) {
            w32[i] = (float)wi;
            aux[2 + i] = (w != nullptr) ? wi * fma(2.0, part, ai[i] * wi) : 0.0;
            aux[2 + n + i] = (w != nullptr) ? wi * mi : 0.0;
        }
    }
    if (bad) atomicExch(info, -1);
}

// The previous panel (columns k0 .. k0 + kb - 1, kb = 0 before the first
// block) applied to the trailing lower triangle, whose first row is
// r0 = k0 + kb, beside CTA 0, which factors the 32 x 32 diagonal block at r0
// (the panel's kernel has brought it up to date) and leaves its reciprocal
// pivots in dinv.
__global__ void __launch_bounds__(kCholCta, 1) chol_step_kernel(double *L, int n, int k0, int kb, double *dinv, int *info)
{
    __shared__ double P[kCholTile][kCholNb + 1];
    __shared__ double col[kCholNb * kCholNb];
    __shared__ double T[kCholTile][kCholNb + 1];
    __shared__ double inv[kCholNb];
    __shared__ CholFlags flags;
    __shared__ int s_fail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r0 = k0 + kb;
    if (blockIdx.x == 0) {
        chol_flags_init(flags);
        if (tid == 0) s_fail = 0;
    }
    pdl_enter();
    if (*info != 0) return;

    if (blockIdx.x > 0) {
        // one 16 x 16 tile (bi, bj), bj <= bi, of the trailing triangle, row
        // by row; tiles 0..2 are the diagonal block's, not touched here
        const int t = (int)blockIdx.x + 2;
        int bi = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f); // then corrected exactly
        while ((bi + 1) * (bi + 2) / 2 <= t) bi++;
        while (bi * (bi + 1) / 2 > t) bi--;
        const int bj = t - bi * (bi + 1) / 2;
        const int i0 = r0 + bi * kCholTile, c0 = r0 + bj * kCholTile;
        // kb == 32 here: a shorter block is the last and has no trailing rows
        for (int e = tid; e < kCholTile * kCholNb; e += blockDim.x) {
            const int r = e / kCholNb, m = e % kCholNb;
            P[r][m] = (i0 + r < n) ? L[(long long)(i0 + r) * n + k0 + m] : 0.0;
            T[r][m] = (c0 + r < n) ? L[(long long)(c0 + r) * n + k0 + m] : 0.0;
        }
        const int r = tid >> 4, c = tid & 15, gi = i0 + r, gj = c0 + c;
        const bool live = gi < n && gj <= gi;
        const double old = live ? L[(long long)gi * n + gj] : 0.0;
        __syncthreads();
        double v = 0.0;
#pragma unroll
        for (int m = 0; m < kCholNb; m++) v = fma(P[r][m], T[c][m], v);
        if (live) L[(long long)gi * n + gj] = old - v;
        return;
    }

    const int nb = min(kCholNb, n - r0);
    for (int e = tid; e < kCholNb * kCholNb; e += blockDim.x) {
        const int r = e / kCholNb, m = e % kCholNb;
        col[m * kCholNb + r] = (r < nb && m <= r) ? L[(long long)(r0 + r) * n + r0 + m] : 0.0;
    }
    __syncthreads();
    if (chol_takes_part()) chol_factor_cta<kCholNb, false>(nb, col, inv, flags, &s_fail);
    __syncthreads();
    if (s_fail) {
        if (tid == 0) *info = s_fail < 0 ? kCholTimeout : r0 + s_fail;
        return;
    }
    for (int e = tid; e < kCholNb * kCholNb; e += blockDim.x) {
        const int r = e / kCholNb, m = e % kCholNb;
        if (r < nb && m <= r) L[(long long)(r0 + r) * n + r0 + m] = col[m * kCholNb + r];
    }
    if (tid < nb) dinv[tid] = inv[tid];
}

// Rows below the diagonal block at k0 (32 columns): x L_kk^T = a, one warp
// per row, lane j holding column j.  With l'_jc = l_jc / l_jj and
// s_j = a_j / l_jj the solve is s_j -= x_c l'_jc for c < j, x_j = s_j: one
// shuffle and one FMA a step.
//
// The 32 rows of cluster 0 are those of the next diagonal block, and it goes
// on to subtract their products from that block: each row is handed to all
// eight CTAs, and 17 warps take a unit of the lower triangle each, two a CTA
// (one SM's FP64 pipe needs 10k cycles for the block; in the factoring CTA
// they stood before the chain of pivots).  The cluster's barriers stand where
// every thread passes them.
static constexpr int kPanelWarps = 4;
static constexpr int kPanelCluster = kCholNb / kPanelWarps;
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__global__ void __cluster_dims__(kPanelCluster, 1, 1) __launch_bounds__(32 * kPanelWarps)
    chol_panel_kernel(double *L, int n, int k0, const double *dinv, const int *info)
{
    __shared__ double lp[kCholNb][kCholNb + 1];
    __shared__ double X[kCholNb][kCholNb + 1]; // cluster 0: the rows of the next diagonal block
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)blockIdx.x; // rank: in cluster 0
    const bool next = blockIdx.x < kPanelCluster;
    pdl_enter();
    if (*info != 0) return; // the same in every CTA
    if (next) cluster_arrive(); // this CTA runs: its X may be written
    const double di = dinv[lane];
    for (int j = warp; j < kCholNb; j += kPanelWarps) {
        const double dj = __shfl_sync(0xffffffffu, di, j);
        lp[j][lane] = lane < j ? L[(long long)(k0 + j) * n + k0 + lane] * dj : 0.0;
    }
    const int r1 = k0 + kCholNb, i = r1 + (int)blockIdx.x * kPanelWarps + warp;
    double s = i < n ? L[(long long)i * n + k0 + lane] * di : 0.0;
    // Unit u of the block's lower triangle: column u (rows u..31) and, in the
    // lanes left over, column 32 - u (rows 32 - u..31): 17 full-width units
    // are half the warp FMAs of the square.
    const int u = warp < 2 ? rank + kPanelCluster * warp : kCholNb / 2;
    const bool unit = next && (warp < 2 || (warp == 2 && rank == 0)) && (u < kCholNb / 2 || lane < kCholNb / 2);
    const int row = lane < kCholNb - u ? u + lane : lane, cc = lane < kCholNb - u ? u : kCholNb - u;
    const bool live = unit && r1 + row < n;
    double *out = L + (live ? (long long)(r1 + row) * n + r1 + cc : 0);
    const double old = live ? *out : 0.0;
    __syncthreads();
    if (i < n || next) {
#pragma unroll
        for (int c = 0; c < kCholNb - 1; c++) {
            const double x = __shfl_sync(0xffffffffu, s, c);
            const double t = fma(-x, lp[lane][c], s);
            s = lane > c ? t : s;
        }
        if (i < n) L[(long long)i * n + k0 + lane] = s;
    }
    if (!next) return;
    cluster_wait();
    const unsigned at = chol_smem(&X[rank * kPanelWarps + warp][lane]);
#pragma unroll
    for (int r = 0; r < kPanelCluster; r++) {
        unsigned remote;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(r));
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote), "d"(s) : "memory");
    }
    cluster_arrive();
    cluster_wait();
    if (!live) return;
    double v = 0.0;
#pragma unroll
    for (int m = 0; m < kCholNb; m++) v = fma(X[row][m], X[cc][m], v);
    *out = old - v;
}

// Packed FP32 rows, and the moment sums in a fixed order (one CTA reduces).
__global__ void chol_finish_kernel(const double *L, int n, float *Lp, double *aux, const int *info)
{
    __shared__ double red[33];
    pdl_enter();
    if (*info != 0) return;
    // one warp per row
    const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
        const int off = packed_row_offset(i), len = 4 * (i / 4 + 1);
        for (int j = lane; j < len; j += 32) Lp[off + j] = (j <= i) ? (float)L[(long long)i * n + j] : 0.f;
    }
    if (blockIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            a += aux[2 + i];
            b += aux[2 + n + i];
        }
        const double wsw = block_sum(a, red);
        const double wmu = block_sum(b, red);
        if (threadIdx.x == 0) {
            aux[0] = wsw;
            aux[1] = wmu;
        }
    }
}

// Launch behind the kernel before it in the stream, without waiting for that
// one to drain (the kernels wait in pdl_enter).
template <class... P, class... A>
static cudaError_t launch_pdl(void (*kern)(P...), int grid, int threads, size_t smem, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

// aux: 2 moments, then 2 n per-row terms, then 32 reciprocal pivots.
static cudaError_t launch_cholesky_blocked(const double *A, long long lda, int n, const double *w,
                                           const double *mu, double *L64, float *Lp, float *w32,
                                           double *aux, int *info, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(info, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
    double *dinv = aux + 2 + 2 * (size_t)n;
    e = cudaFuncSetAttribute(chol_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCholAlone);
    if (e != cudaSuccess) return e;
    chol_prep_kernel<<<(n + 7) / 8, 256, 0, s>>>(A, lda, n, w, mu, L64, w32, aux, info);
    e = cudaGetLastError();
    for (int k0 = 0, kb = 0; e == cudaSuccess && k0 + kb < n;) {
        const int r0 = k0 + kb, nt = (n - r0 + kCholTile - 1) / kCholTile;
        const int tiles = (kb > 0 && nt > 2) ? nt * (nt + 1) / 2 - 3 : 0;
        // While the factoring CTA is the longest, it keeps its SM's FP64 pipe
        // to itself (shared memory for one CTA an SM); with more than about
        // six tiles an SM the trailing update is, and packs the SMs.
        const size_t alone = tiles <= 6 * kSms ? kCholAlone : 0;
        e = launch_pdl(chol_step_kernel, 1 + tiles, kCholCta, alone, s, L64, n, k0, kb, dinv, info);
        k0 = r0;
        kb = n - r0 < kCholNb ? n - r0 : kCholNb;
        const int rest = n - k0 - kb;
        if (e == cudaSuccess && rest > 0)
            e = launch_pdl(chol_panel_kernel, (rest + kCholNb - 1) / kCholNb * kPanelCluster, 32 * kPanelWarps, 0, s, L64,
                           n, k0, (const double *)dinv, (const int *)info);
    }
    if (e != cudaSuccess) return e;
    return launch_pdl(chol_finish_kernel, (n + 7) / 8, 256, 0, s, (const double *)L64, n, Lp, aux, (const int *)info);
}

int cholesky_max_n() { return kCholMaxN; }

// aux holds cholesky_aux_len(n) doubles: the two moments, then scratch.
size_t cholesky_aux_len(int n) { return 2 + 2 * (size_t)n + kCholNb; }

cudaError_t launch_cholesky(const double *A, long long lda, int n, const double *w,
                            const double *mu, double *L64, float *Lp, float *w32, double *aux,
                            int *info, cudaStream_t s)
{
    if (n > kCholMaxN) return cudaErrorInvalidValue;
    // RG_CHOLESKY=single|blocked overrides the size rule (for tests)
    const char *sel = getenv("RG_CHOLESKY");
    bool blocked = n > kCholSmallMaxN;
    if (sel && strstr(sel, "single")) blocked = false;
    if (sel && strstr(sel, "blocked")) blocked = true;
    if (blocked) return launch_cholesky_blocked(A, lda, n, w, mu, L64, Lp, w32, aux, info, s);
    if (n <= kCholSmallMaxN) {
        // NC in steps of 16: columns between n and NC cost their multiply-adds
        auto kern = n <= 16 ? chol_small_kernel<16> : n <= 32 ? chol_small_kernel<32> : n <= 48 ? chol_small_kernel<48>
                                                                                               : chol_small_kernel<64>;
        kern<<<1, kCholCta, 0, s>>>(A, lda, n, w, mu, L64, Lp, w32, aux, info);
        return cudaGetLastError();
    }
    const size_t smem = sizeof(double) * (size_t)(n > 0 ? n : 1);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(cholesky_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return e;
    }
    cholesky_kernel<<<1, kCholThreads, smem, s>>>(A, lda, n, w, mu, L64, Lp, w32, aux, info);
    return cudaGetLastError();
}

} // namespace rg
