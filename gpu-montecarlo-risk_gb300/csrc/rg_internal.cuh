// Internal declarations shared by the engine's translation units.
//
// Device helpers:
//   rg_philox       Philox4x32-10 (Salmon et al., SC'11): 10 rounds of two
//                   32x32->64 multiplies with the published multipliers and
//                   Weyl key increments.  Round keys are precomputed on the
//                   host (they depend only on the seed).
//   rg_box_muller   Box-Muller (Box & Muller 1958) on two 32-bit words.
//                   The top 23 bits of a word w form f = 1 + (w >> 9) 2^-23 in
//                   [1, 2) by setting the exponent bits (no int->float
//                   conversion); u_a = 2 - f in (0, 1], t = 2 pi f_b in
//                   [2 pi, 4 pi) (a uniform angle), r = sqrt(-2 ln u_a),
//                   (z0, z1) = (r cos t, r sin t), using the hardware
//                   approximate lg2/sqrt/sin/cos (PTX *.approx).  The
//                   smallest u_a is 2^-23, so |z| <= sqrt(46 ln 2) = 5.65.
#pragma once

#include <cstdint>
#include <atomic>
#include <vector>
#include <cuda_runtime.h>

#include "riskgpu.h"

namespace rg {

// ---------------------------------------------------------------- device
struct PhiloxKeys {
    uint32_t k0[10];
    uint32_t k1[10];
};

inline PhiloxKeys philox_round_keys(uint64_t seed)
{
    PhiloxKeys k;
    uint32_t a = (uint32_t)seed, b = (uint32_t)(seed >> 32);
    for (int r = 0; r < 10; r++) {
        k.k0[r] = a;
        k.k1[r] = b;
        a += 0x9E3779B9u;
        b += 0xBB67AE85u;
    }
    return k;
}

__device__ __forceinline__ uint4 rg_philox(uint4 c, const PhiloxKeys &k)
{
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * c.x;
        const uint64_t p1 = (uint64_t)0xCD9E8D57u * c.z;
        const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
        const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
        c = make_uint4(hi1 ^ c.y ^ k.k0[r], lo1, hi0 ^ c.w ^ k.k1[r], lo0);
    }
    return c;
}

// Two independent Philox4x32-10 blocks, rounds interleaved (the same words
// as two rg_philox calls; more independent work per thread where few warps
// share an SM).
__device__ __forceinline__ void rg_philox2(uint4 &a, uint4 &b, const PhiloxKeys &k)
{
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * a.x, p1 = (uint64_t)0xCD9E8D57u * a.z;
        const uint64_t q0 = (uint64_t)0xD2511F53u * b.x, q1 = (uint64_t)0xCD9E8D57u * b.z;
        a = make_uint4((uint32_t)(p1 >> 32) ^ a.y ^ k.k0[r], (uint32_t)p1, (uint32_t)(p0 >> 32) ^ a.w ^ k.k1[r],
                       (uint32_t)p0);
        b = make_uint4((uint32_t)(q1 >> 32) ^ b.y ^ k.k0[r], (uint32_t)q1, (uint32_t)(q0 >> 32) ^ b.w ^ k.k1[r],
                       (uint32_t)q0);
    }
}

// The first two rounds of Philox4x32-10 for counter (block, 0, lo, hi), split
// by what they depend on.  With hi1(.), lo1(.) the halves of 0xCD9E8D57 x and
// hi0, lo0 those of 0xD2511F53 x, the state after round 2 is
//   x = hi1(hi0(block) ^ hi ^ k1[0]) ^ k0[1]  ^  lo1(lo)
//   y = lo1(hi0(block) ^ hi ^ k1[0])
//   z = hi0(hi1(lo) ^ k0[0])  ^  lo0(block) ^ k1[1]
//   w = lo0(hi1(lo) ^ k0[0])
// so for path indexes with the same high word, the left term of x, y and the
// right term of z belong to the block alone (PhiloxBlock, with round 3's k0
// folded into y; a table over a query's blocks is laid out once per launch)
// and the rest to the path (PhiloxPath, with round 3's k1 folded into w).
// A block of four words then costs 16 wide multiplies instead of 18; each
// takes 4.2 cycles of one multiplier pipe per SM sub-partition (measured),
// the busiest pipe of Philox.
struct __align__(16) PhiloxBlock {
    uint32_t x, y, z, pad;
};
struct PhiloxPath {
    uint32_t x, z, w;
};
__host__ __device__ __forceinline__ PhiloxBlock philox_block(uint32_t block, uint32_t hi, const PhiloxKeys &k)
{
    const uint64_t p = (uint64_t)0xD2511F53u * block;
    const uint64_t q = (uint64_t)0xCD9E8D57u * ((uint32_t)(p >> 32) ^ hi ^ k.k1[0]);
    PhiloxBlock b;
    b.x = (uint32_t)(q >> 32) ^ k.k0[1];
    b.y = (uint32_t)q ^ k.k0[2];
    b.z = (uint32_t)p ^ k.k1[1];
    b.pad = 0u;
    return b;
}
__device__ __forceinline__ PhiloxPath philox_path(uint32_t lo, const PhiloxKeys &k)
{
    const uint64_t q = (uint64_t)0xCD9E8D57u * lo;
    const uint64_t p = (uint64_t)0xD2511F53u * ((uint32_t)(q >> 32) ^ k.k0[0]);
    PhiloxPath c;
    c.x = (uint32_t)q;
    c.z = (uint32_t)(p >> 32);
    c.w = (uint32_t)p ^ k.k1[2];
    return c;
}
// State after round 3 (of 10).
__device__ __forceinline__ uint4 philox_join(const uint4 &b, const PhiloxPath &c)
{
    const uint64_t p0 = (uint64_t)0xD2511F53u * (b.x ^ c.x);
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * (b.z ^ c.z);
    return make_uint4((uint32_t)(p1 >> 32) ^ b.y, (uint32_t)p1, (uint32_t)(p0 >> 32) ^ c.w, (uint32_t)p0);
}
// The words of two blocks of one path, rounds interleaved: the same as
// rg_philox2 on their counters.
__device__ __forceinline__ void rg_philox2_from(const uint4 &ta, const uint4 &tb, const PhiloxPath &path,
                                                const PhiloxKeys &k, uint4 &a, uint4 &b)
{
    a = philox_join(ta, path);
    b = philox_join(tb, path);
#pragma unroll
    for (int r = 3; r < 10; r++) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * a.x, p1 = (uint64_t)0xCD9E8D57u * a.z;
        const uint64_t q0 = (uint64_t)0xD2511F53u * b.x, q1 = (uint64_t)0xCD9E8D57u * b.z;
        a = make_uint4((uint32_t)(p1 >> 32) ^ a.y ^ k.k0[r], (uint32_t)p1, (uint32_t)(p0 >> 32) ^ a.w ^ k.k1[r],
                       (uint32_t)p0);
        b = make_uint4((uint32_t)(q1 >> 32) ^ b.y ^ k.k0[r], (uint32_t)q1, (uint32_t)(q0 >> 32) ^ b.w ^ k.k1[r],
                       (uint32_t)q0);
    }
}

__device__ __forceinline__ float rg_lg2_approx(float x)
{
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rg_sqrt_approx(float x)
{
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rg_sin_approx(float x)
{
    float y;
    asm("sin.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rg_cos_approx(float x)
{
    float y;
    asm("cos.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// 1 + (w >> 9) 2^-23, exactly, in [1, 2)
__device__ __forceinline__ float rg_one_to_two(uint32_t w)
{
    return __uint_as_float(0x3f800000u | (w >> 9));
}

__device__ __forceinline__ void rg_box_muller(uint32_t a, uint32_t b, float &z0, float &z1)
{
    const float ua = 2.0f - rg_one_to_two(a);          // (0, 1]
    // -2 ln(u) = -2 ln(2) log2(u)
    const float r = rg_sqrt_approx(-1.3862943611198906f * rg_lg2_approx(ua));
    const float t = 6.283185307179586f * rg_one_to_two(b); // [2 pi, 4 pi)
    z0 = r * rg_cos_approx(t);
    z1 = r * rg_sin_approx(t);
}

// sqrt(2 ln 2): r = sqrt(-2 ln u) = kBmScale sqrt(-log2 u).
static constexpr float kBmScale = 1.1774100225154747f;

// Box-Muller as above without the factor sqrt(2 ln 2) of r: returns
// (z0, z1) / sqrt(2 ln 2), one multiply fewer a pair.  For callers that sum
// several draws and scale the sum once.
__device__ __forceinline__ void rg_box_muller_unscaled(uint32_t a, uint32_t b, float &z0, float &z1)
{
    const float ua = 2.0f - rg_one_to_two(a);          // (0, 1]
    const float r = rg_sqrt_approx(-rg_lg2_approx(ua));
    const float t = 6.283185307179586f * rg_one_to_two(b); // [2 pi, 4 pi)
    z0 = r * rg_cos_approx(t);
    z1 = r * rg_sin_approx(t);
}

// Packed FP32 lower-triangular rows: row i holds L[i][0..i] zero-padded to
// a multiple of 4 floats, so every row starts on a 16-byte boundary.
// offset(i) = sum_{r<i} 4 ceil((r+1)/4) = 4 (a+1)(2a+b) for i = 4a+b.
__host__ __device__ constexpr int packed_row_offset(int i)
{
    return 4 * (i / 4 + 1) * (2 * (i / 4) + (i % 4));
}
__host__ __device__ constexpr int packed_len(int n) { return packed_row_offset(n); }

// SMs of a GB300, for splits of work whose order of sums must not depend on the
// device that runs them (launch grids take the device's own count).
static constexpr int kSms = 152;

// ---------------------------------------------------------------- host
struct Portfolio {
    int n = 0;
    int has_w = 0;
    int device = 0;
    bool pooled = false;       // d_block is from the engine's pool (else from cudaMalloc)
    size_t block_bytes = 0;
    // Work that no call of the engine waits for may read d_block: a launch on a
    // caller's stream, a batch or a server, or the caller's own (its pointers
    // were handed out).  Set by every entry point that lets that happen.
    mutable std::atomic<bool> shared{false};
    void *d_block = nullptr;   // one allocation holding every device buffer below
    double *d_L64 = nullptr;   // n x n row-major, zero upper
    double *d_mu64 = nullptr;  // n
    float *d_Lp = nullptr;     // packed rows (packed_len(n) floats)
    float *d_Lt = nullptr;     // L^T FP32 [tiled_kpad(n)][tiled_npad(n)], zero padded
    unsigned char *d_tc[2] = {nullptr, nullptr}; // tensor-core tiles (FP16, BF16), N <= tc_max_n()
    unsigned int *d_err = nullptr; // error word of the tensor-core kernel
    float *d_w32 = nullptr;    // n (zeros when no weights)
    double *d_aux = nullptr;   // w^T Sigma w, w.mu, then scratch of the factorisation and the tile build
    int *d_info = nullptr;
    double wsw = 0.0, wmu = 0.0;
    float ms_chol = 0.f;
    // N <= 64: host copies for the kernel that takes the factor by value
    std::vector<float> h_Lp;   // packed rows, FP32
    std::vector<double> h_mu;  // daily means, FP64
    std::vector<float> h_w;    // weights, FP32 (zeros when none)
};

// Counters of one query.  Kernels add to the device copy; with PlainArgs::head
// set, the last CTA of a launch writes them to `host` and resets them.
struct QueryHead {
    unsigned long long counts[2];  // crash, breach
    unsigned long long tail[2];    // VaR tail: paths, sum of -w.R * 2^32 (int64 bits)
    unsigned int cand_count;       // VaR candidates
    unsigned int err;              // error word of the tensor-core kernel
    unsigned int ctas;             // CTAs that are done (device)
    unsigned int pad[5];
};
static_assert(sizeof(QueryHead) == 64, "read in 8-byte words");

// Arguments of the fused counting kernels.
struct PlainArgs {
    const float4 *Lp;
    const double *mu64;
    const float *w;
    int n;
    int horizon;
    long long n_paths;
    unsigned long long path0;
    unsigned long long seed;
    PhiloxKeys keys;
    float neg_x;
    float port_thr;
    int k;
    int has_w;
    int aggregated;            // draw mode RG_DRAWS_AGGREGATED
    int *s_values;
    float *port_values;
    unsigned long long *counts; // [2]
    // VaR / CVaR passes (kernels instantiated with VaR support only).
    // Every path's portfolio return w.R falls in bin
    //   b = floor((w.R - sel_lo) * sel_inv_w), clamped to [-1, sel_bins].
    // var_mode 1 (select): b < sel_target -> tail (count, fixed-point loss
    //   sum); b == sel_target -> candidate appended to cand[].
    // var_mode 2 (histogram): counts per bin into hist[sel_bins + 2].
    int var_mode;
    int sel_bins;
    int sel_target;
    float sel_lo;
    float sel_inv_w;
    float *cand;
    unsigned int *cand_count;
    unsigned int cand_cap;
    unsigned long long *tail;   // [0] tail paths, [1] sum of -w.R * 2^32 (int64 bits)
    unsigned long long *hist;   // [sel_bins + 2]
    unsigned int *err;          // device error word of the tensor-core kernel (bounded waits)
    QueryHead *head;            // device counters to report and reset, or null
    QueryHead *host;            // pinned host memory they are reported to
    // room for the query's PhiloxBlock table (philox_table_len entries), or null
    PhiloxBlock *blocks;
};

// End of a launch for one thread of each CTA, after every count of its CTA has
// been added (a CTA barrier before it).  The CTA that is last reports the
// query's counters to pinned host memory and leaves zeros for the next launch.
__device__ __forceinline__ void cta_report(const PlainArgs &a)
{
    if (!a.head) return;
    __threadfence();
    if (atomicAdd(&a.head->ctas, 1u) != gridDim.x - 1u) return;
    __threadfence();
    unsigned long long *d = reinterpret_cast<unsigned long long *>(a.head);
    volatile unsigned long long *h = reinterpret_cast<volatile unsigned long long *>(a.host);
    unsigned long long v[sizeof(QueryHead) / 8];
#pragma unroll
    for (int i = 0; i < (int)(sizeof(QueryHead) / 8); i++) v[i] = __ldcg(d + i);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(QueryHead) / 8); i++) {
        h[i] = v[i];
        d[i] = 0ull;
    }
    __threadfence_system();
}

// Entries of a query's block table (block = day * ceil(N/4) + quad), or 0
// where it is not used: the paths' high words differ or the table is longer
// than 1 MiB.
inline size_t philox_table_len(int n, int days, unsigned long long path0, long long n_paths)
{
    const unsigned long long last = path0 + (unsigned long long)(n_paths - 1);
    const size_t len = (size_t)((n + 3) / 4) * (size_t)days;
    return (path0 >> 32) == (last >> 32) && len <= 65536 ? len : 0;
}

// Shared-memory histogram size of the VaR pass: bins plus under/overflow.
static constexpr int kVarHistBins = 4096;

// Launchers.  Return cudaSuccess or the launch error.
// Fills a query's block table (rg_mc_tc.cu).
cudaError_t launch_philox_table(PhiloxBlock *t, size_t len, unsigned long long path0, const PhiloxKeys &keys,
                                cudaStream_t s);
// rg_mc_plain.cu / rg_mc_xorwow.cu: row-order kernel, L staged in shared
// memory; both normal layouts.
cudaError_t launch_plain_small(const PlainArgs &a, int rng, int sm_count, cudaStream_t s);
int plain_small_max_n();
// rg_mc_tiled.cu: general-N tiled kernel (Philox layout).
cudaError_t launch_tiled(const PlainArgs &a, const float *Lt, bool aggregated, int sm_count,
                         cudaStream_t s);
cudaError_t launch_build_lt(const double *L64, int n, float *Lt, cudaStream_t s);
int tiled_max_n();
int tiled_npad(int n);
int tiled_kpad(int n);
// rg_mc_tc.cu: tcgen05 precision form (Philox layout), N <= tc_max_n().
cudaError_t launch_tc(const PlainArgs &a, const unsigned char *tiles, int bf16, bool aggregated, double wmu,
                      unsigned int *err, bool inject_stall, int sm_count, cudaStream_t s);
// the tensor tiles of either split (null: not wanted); scratch: tc_scratch_len(n) doubles
cudaError_t launch_build_tc_tiles(const double *L64, const float *w32, int n, double *scratch, unsigned char *fp16,
                                  unsigned char *bf16, cudaStream_t s);
size_t tc_scratch_len(int n);
int tc_max_n();
size_t tc_tile_bytes(int n);
// batches of (portfolio, query) items in one persistent launch (a.blocks: room
// for the item's block table, filled by launch_batch_tables, or null)
cudaError_t launch_batch_tables(const void *d_items, int count, cudaStream_t s);
void tc_fill_batch_item(void *item_out, const PlainArgs &a, const unsigned char *tiles, int bf16,
                        bool aggregated, double wmu, long long tile_begin);
size_t tc_item_bytes();
long long tc_tiles_of(long long n_paths, int paths_per_tile);
int tc_batch_paths(int n_mt_max);
int tc_row_tiles_of(int n);
int tc_k_tiles_of(int n);
cudaError_t launch_tc_batch(const void *d_items, int n_items, long long total_tiles, int unit_tiles,
                            unsigned int *work, unsigned int *err, int n_kt_max, int n_mt_max, bool split, int grid,
                            cudaStream_t s, const long long *dyn = nullptr);
int tc_max_k_tiles();
double tc_tile_gen(int n, int days, int paths);
double tc_tile_mma(int n);
bool tc_split_wins(double gen, double mma);
cudaError_t tc_batch_prepare();
int tc_batch_occupancy(int n_mt_max);
// rg_mc_fused.cu: N <= 64 kernel, L in parameter space; Philox only.
cudaError_t launch_fused(const PlainArgs &a, const float *Lp_host, const float *hmu, const float *w,
                         int sm_count, cudaStream_t s);
int fused_max_n();

// Cholesky (rg_cholesky.cu): factor, pack and portfolio moments.
cudaError_t launch_cholesky(const double *A, long long lda, int n, const double *w,
                            const double *mu, double *L64, float *Lp, float *w32, double *aux,
                            int *info, cudaStream_t s);
int cholesky_max_n();
size_t cholesky_aux_len(int n);

// Error helpers (rg_capi.cu).
int set_error(int status, const char *fmt, ...);

// Stream-ordered device memory from the engine's pool of the current device
// (rg_capi.cu; freed with cudaFreeAsync).  Returns RG_OK with *err the
// allocation's result, or the status of a device that could not be set up.
int pool_alloc(void **p, size_t bytes, cudaStream_t s, cudaError_t *err);
void pool_trim();
// Whether the free-memory admission check would let `need` bytes through (for
// memory that a call can do without).
bool admits(size_t need);
// cudaMalloc, tried once more after pool_trim.
cudaError_t device_alloc(void **p, size_t bytes);
template <class T> inline cudaError_t device_alloc(T **p, size_t bytes)
{
    return device_alloc(reinterpret_cast<void **>(p), bytes);
}

} // namespace rg
