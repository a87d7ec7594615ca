// Operand preparation of the modular contraction: row scales and BF16 residue planes
// (sm_103a).  Included by the translation units that name an operand source.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "digits.cuh"
#include "modular.cuh"
#include "moduli.cuh"
#include "tc.cuh"

namespace cutc {

// ---------------------------------------------------------------------------
// operand sources: value of row r, column k of an FP64 matrix, and up(r, k) >= its
// magnitude as a float (within 2^-21; 0 below the float range, infinity above it, NaN
// for a NaN)
// ---------------------------------------------------------------------------

__device__ __forceinline__ float abs_up(double x)
{
    // from the high word, with integer operations: FP64 conversions take the FP64 pipe
    const int hi = __double2hiint(x) & 0x7fffffff;
    if (hi >= 0x7ff00000)
        return __int_as_float(0x7fffffff);
    const int v = hi - 0x38000000;  // exponent bias 1023 -> 127
    if (v < 0x00100000)
        return 0.0f;
    if (v >= 0x0fe00000)
        return __int_as_float(0x7f800000);
    return __int_as_float((v << 3) + 8);
}

struct SrcDense {  // X[r * ld + k]
    static constexpr bool kDoubleFloat = false;
    const double *X;
    int64_t ld;
    __device__ double operator()(int64_t r, int64_t k) const { return X[r * ld + k]; }
    __device__ float up(int64_t r, int64_t k) const { return abs_up(X[r * ld + k]); }
};

struct SrcConcat {  // [X1 | X2]: X1[r * k1 + k] for k < k1, then X2[r * k2 + k - k1]
    static constexpr bool kDoubleFloat = false;
    const double *X1, *X2;
    int64_t k1, k2;
    __device__ double operator()(int64_t r, int64_t k) const
    {
        return k < k1 ? X1[r * k1 + k] : X2[r * k2 + (k - k1)];
    }
    __device__ float up(int64_t r, int64_t k) const { return abs_up((*this)(r, k)); }
};

struct SrcDenseDF {  // hi + lo of X[r * ld + k]; the residues are cut from the pair itself
    static constexpr bool kDoubleFloat = true;
    const float2 *X;
    int64_t ld;
    __device__ float2 pair(int64_t r, int64_t k) const { return X[r * ld + k]; }
    __device__ double operator()(int64_t r, int64_t k) const
    {
        const float2 v = X[r * ld + k];
        return (double)v.x + (double)v.y;
    }
    __device__ float up(int64_t r, int64_t k) const
    {
        return fabsf(X[r * ld + k].x) * 1.0000002f;
    }
};

// The pair products take their first factor w chi_a from a table of the weighted AO
// rows, formed once per AO (weighted_aos_kernel) instead of once per pair: FP64
// multiplies run at 1/64 of the FP32 rate on GB300.
struct SrcSym {  // w[k] chi_a(k) chi_b(k) = (w chi_a)(k) chi_b(k), (a, b) = pairs[r]
    static constexpr bool kDoubleFloat = false;
    const double *wchi, *chi;  // wchi[a * K + k] = w[k] chi_a(k); chi_b at chi[b * ldchi + k]
    int64_t K, ldchi;
    const int2 *pairs;
    __device__ double operator()(int64_t r, int64_t k) const
    {
        const int2 ab = pairs[r];
        return wchi[ab.x * K + k] * chi[ab.y * ldchi + k];
    }
    __device__ float up(int64_t r, int64_t k) const
    {
        const int2 ab = pairs[r];
        return abs_up(wchi[ab.x * K + k]) * abs_up(chi[ab.y * ldchi + k]);
    }
};

// w (chi_c d_m chi_d - chi_d d_m chi_c) as (w chi_c) d_m chi_d - (w chi_d) d_m chi_c,
// k = m n + g, (c, d) = pairs[r]
struct SrcAnti {
    static constexpr bool kDoubleFloat = false;
    const double *wchi, *aos;  // wchi[c * n + g] = w[g] chi_c(g); aos: (ld, nA, 4) with
                               // the grid offset already applied
    int n, nA;                 // n: grid points counted in k (g < n)
    int64_t ld;                // grid stride of aos
    const int2 *pairs;
    __device__ double operator()(int64_t r, int64_t k) const
    {
        int m, g;
        if (k < 0x7fffffff) {  // 32-bit division (K = 3 n)
            const unsigned ku = (unsigned)k, mu = ku / (unsigned)n;
            m = (int)mu;
            g = (int)(ku - mu * (unsigned)n);
        } else {
            m = (int)(k / n);
            g = (int)(k % n);
        }
        const int2 cd = pairs[r];
        const int64_t comp = (int64_t)nA * ld * (m + 1);
        return fma(wchi[(int64_t)cd.x * n + g], aos[comp + cd.y * ld + g],
                   -(wchi[(int64_t)cd.y * n + g] * aos[comp + cd.x * ld + g]));
    }
    __device__ float up(int64_t r, int64_t k) const { return abs_up((*this)(r, k)); }
};

// ---------------------------------------------------------------------------
// row scales
// ---------------------------------------------------------------------------

// |v| as its bits (non-negative doubles order like their bits)
__device__ __forceinline__ unsigned long long abs_bits(double v)
{
    return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}

// The scale of a row of norm sqrt(ss) 2^e: floor(bits - log2 |row|_2), with the sum's even
// power of two taken out first, so that a row times a power of two has the same digits.  The
// 0.0005 covers the rounding of the sum (up to 2^20 columns in FP32).
__device__ __forceinline__ int norm_scale(float ss, float bits, int e)
{
    const int b = __float_as_int(ss);
    const int j = ((b >> 23) - 127) >> 1;
    const float f = __int_as_float(b - j * (1 << 24));  // ss 4^-j, in [1, 4)
    return (int)floorf(bits - 0.5f * log2f(f) - 0.0005f) - j - e;
}

constexpr int64_t kFloatSums = 1 << 20;  // columns up to which FP32 sums do

// ... from the row's maximum m and sum of squares ss in FP32 when both are well inside the
// float range.
__device__ __forceinline__ bool scale_fast(float m, float ss, float bits, int64_t K, int *s)
{
    if (K > kFloatSums || !(m >= 0x1p-50f && m <= 0x1p60f && ss <= 0x1p125f))
        return false;
    *s = norm_scale(ss, bits, 0);
    return true;
}

// Other rows (values near the ends of the FP64 range, long rows) are summed a second time,
// scaled by their largest |x|, given as bits: e with |x| < 2^e.
__device__ __forceinline__ int max_exponent(unsigned long long mb)
{
    const int E = (int)(mb >> 52);  // (a subnormal's leading bit counts from 2^-1074)
    return E ? E - 1022 : mb ? -1010 - __clzll((long long)mb) : 0;
}

__device__ __forceinline__ float scaled_up(double x, int e) { return abs_up(scalbn(x, -e)); }

// ... and their scale: ss is that sum.  Zero rows have scale 0, rows with an infinity or a NaN
// kNotFinite.
__device__ __forceinline__ int scale_slow(unsigned long long mb, float ss, float bits)
{
    if ((int)(mb >> 52) >= 0x7ff)
        return kNotFinite;
    return mb ? norm_scale(ss, bits, max_exponent(mb)) : 0;
}

// The sum of v over the block's 256 threads, in a fixed order, for thread 0.
template <class T>
__device__ __forceinline__ T block_sum(T v, T (&part)[8])
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();  // the previous values are read
    if ((threadIdx.x & 31) == 0)
        part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < 8; w++)
            v += part[w];
    return v;
}

// sc[r] for every row: one block per row (a fixed summation order, so the scale never
// depends on scheduling); reads the row once.
template <class Src>
__global__ void __launch_bounds__(256)
row_scale_kernel(Src src, int rows, int64_t K, float bits, int *__restrict__ sc)
{
    __shared__ float sm[8], sq[8];
    __shared__ double sd[8];
    __shared__ unsigned long long sb[8], s_max;
    __shared__ int s_fast;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        float m = 0.0f, ss = 0.0f;
#pragma unroll 4
        for (int64_t k = threadIdx.x; k < K; k += 256) {
            const float v = src.up(r, k);
            m = fmaxf(m, v);
            ss = fmaf(v, v, ss);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0)
            sm[warp] = m;  // (read below before the next row's, behind block_sum's barriers)
        ss = block_sum(ss, sq);
        if (threadIdx.x == 0) {
            for (int w = 1; w < 8; w++)
                m = fmaxf(m, sm[w]);
            int s = 0;
            s_fast = scale_fast(m, ss, bits, K, &s);
            if (s_fast)
                sc[r] = s;
        }
        __syncthreads();
        if (s_fast)
            continue;
        unsigned long long mb = 0;
        for (int64_t k = threadIdx.x; k < K; k += 256) {
            const unsigned long long b = abs_bits(src(r, k));
            mb = b > mb ? b : mb;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long b = __shfl_xor_sync(0xffffffffu, mb, o);
            mb = b > mb ? b : mb;
        }
        if (lane == 0)
            sb[warp] = mb;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < 8; w++)
                mb = sb[w] > mb ? sb[w] : mb;
            s_max = mb;
        }
        __syncthreads();
        mb = s_max;
        const int e = max_exponent(mb);
        if (K <= kFloatSums) {
            ss = 0.0f;
            for (int64_t k = threadIdx.x; k < K; k += 256) {
                const float v = scaled_up(src(r, k), e);
                ss = fmaf(v, v, ss);
            }
            ss = block_sum(ss, sq);
        } else {
            double s2 = 0.0;
            for (int64_t k = threadIdx.x; k < K; k += 256) {
                const float v = scaled_up(src(r, k), e);
                s2 += (double)v * v;
            }
            ss = (float)block_sum(s2, sd);
        }
        if (threadIdx.x == 0)
            sc[r] = scale_slow(mb, ss, bits);
    }
}

// The magnitude |x| 2^s 2^-kMagnitudeShift as the bits of a BF16 number, truncated (at least
// 2^-60 for x != 0, so that a product of two is not lost); integer arithmetic.
__device__ __forceinline__ unsigned magnitude_bf16(double x, int s)
{
    unsigned long long b = abs_bits(x);
    if (b == 0)
        return 0;
    int E = (int)(b >> 52);
    if (E == 0) {  // subnormal: its leading bit to bit 52
        const int lz = __clzll((long long)b) - 11;
        b <<= lz;
        E = 1 - lz;
    }
    const int e = E - 1023 + s - kMagnitudeShift;
    return (unsigned)(max(e, -60) + 127) << 7 | (e >= -60 ? (unsigned)(b >> 45) & 0x7fu : 0u);
}

// ... of eight values, 16 bytes.
__device__ __forceinline__ void store_magnitudes(const double (&x)[8], int s, __nv_bfloat16 *dst)
{
    unsigned w[4];
#pragma unroll
    for (int q = 0; q < 4; q++)
        w[q] = magnitude_bf16(x[2 * q], s) | magnitude_bf16(x[2 * q + 1], s) << 16;
    *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
}

// The residues of eight integers per thread, chunk[j][q] holding the 13-bit chunks j of
// elements 2q and 2q + 1: every FP32 operation is exact.
template <int N, int CH>
__device__ __forceinline__ void store_residues(const uint64_t (&chunk)[CH][4], __nv_bfloat16 *dst,
                                               int64_t plane)
{
    const uint64_t magic = tc::f2_dup(12582912.0f);  // 1.5 * 2^23: rounds to an integer
#pragma unroll
    for (int i = 0; i < N; i++) {
        unsigned w[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            uint64_t S = chunk[0][q];
#pragma unroll
            for (int j = 1; j < CH; j++)
                S = tc::f2_fma(chunk[j][q], c_tab.chunk[i][j], S);
            const uint64_t d = tc::f2_sub(tc::f2_fma(S, c_tab.inv[i], magic), magic);
            const uint64_t r = tc::f2_fma(d, c_tab.negp[i], S);
            const __nv_bfloat162 v = __floats2bfloat162_rn(tc::f2_lo(r), tc::f2_hi(r));
            w[q] = *reinterpret_cast<const unsigned *>(&v);
        }
        *reinterpret_cast<uint4 *>(dst + i * plane) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// chunk j of the integer rint(x 2^s) as an exact float with the integer's sign
template <int CH>
__device__ __forceinline__ void int_chunks(double x, int s, float (&c)[CH])
{
    using T = std::conditional_t<(CH <= 5), unsigned long long, unsigned __int128>;
    const T a = moduli::scaled_magnitude<T>(x, s);
    const unsigned sign = (unsigned)(__double2hiint(x)) & 0x80000000u;
#pragma unroll
    for (int j = 0; j < CH; j++) {
        const unsigned u = (unsigned)(a >> (moduli::kChunkBits * j)) & 0x1fffu;
        const float f = __uint_as_float(0x4b000000u | u) - 8388608.0f;
        c[j] = __uint_as_float(__float_as_uint(f) ^ sign);
    }
}

template <int N>
__device__ __forceinline__ void pack_chunks(const float (&v)[8][moduli::chunks(N)],
                                            uint64_t (&chunk)[moduli::chunks(N)][4])
{
#pragma unroll
    for (int j = 0; j < moduli::chunks(N); j++)
#pragma unroll
        for (int q = 0; q < 4; q++)
            chunk[j][q] = tc::f2_pack(__float_as_uint(v[2 * q][j]), __float_as_uint(v[2 * q + 1][j]));
}

// An element as its source holds it, a bound of its magnitude, and its 13-bit chunks scaled
// by 2^s.
template <bool DF>
struct ValueOf {
    using T = double;
};
template <>
struct ValueOf<true> {
    using T = float2;
};

template <class Src>
__device__ __forceinline__ typename ValueOf<Src::kDoubleFloat>::T value_of(const Src &src, int64_t r,
                                                                           int64_t k)
{
    if constexpr (Src::kDoubleFloat)
        return src.pair(r, k);
    else
        return src(r, k);
}

__device__ __forceinline__ float up_of(double x) { return abs_up(x); }
__device__ __forceinline__ float up_of(float2 x) { return fabsf(x.x) * 1.0000002f; }

template <int N>
__device__ __forceinline__ void residue_chunks(double x, int s, float (&v)[moduli::chunks(N)])
{
    int_chunks<moduli::chunks(N)>(x, s, v);
}

template <int N>
__device__ __forceinline__ void residue_chunks(float2 x, int s, float (&v)[moduli::chunks(N)])
{
    constexpr int CH = moduli::chunks(N);
    float d[CH];  // from the top: d[0] is chunk CH - 1
    digits::digits_df_fp32<CH, moduli::kChunkBits>(x.x, x.y, moduli::kChunkBits * CH - 1 - s, d);
#pragma unroll
    for (int j = 0; j < CH; j++)
        v[j] = d[CH - 1 - j];
}

// planes[i][r][k - k0] = residues of rint(src(r0 + r, k) 2^{sc[r0 + r]}) modulo p_i for
// rows r < rows and k0 <= k < k0 + kp (zeros up to the row pitch), and with kMag the
// magnitudes as plane N.  Eight consecutive k
// per thread: one 16-byte store per plane.  Bound by the stores: 2 N bytes are written
// per 8-byte element read.
template <int N, bool kMag, class Src>
__global__ void __launch_bounds__(128)
residue_rows_kernel(Src src, int r0, int rows, int64_t k0, int64_t kp, int64_t pitch,
                    const int *__restrict__ sc, __nv_bfloat16 *__restrict__ planes)
{
    constexpr int CH = moduli::chunks(N);
    const int64_t kk = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (kk >= pitch)
        return;
    for (int r = blockIdx.y; r < rows; r += gridDim.y) {
        const int s = max(sc[r0 + r], -4096);  // (kNotFinite: the result is NaN anyway)
        typename ValueOf<Src::kDoubleFloat>::T x[8];
        float v[8][CH];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            x[q] = kk + q < kp ? value_of(src, r0 + r, k0 + kk + q)
                               : typename ValueOf<Src::kDoubleFloat>::T{};
            residue_chunks<N>(x[q], s, v[q]);
        }
        __nv_bfloat16 *dst = planes + (int64_t)r * pitch + kk;
        if constexpr (kMag)
            store_magnitudes(x, s, dst + N * (int64_t)rows * pitch);
        uint64_t chunk[CH][4];
        pack_chunks<N>(v, chunk);
        store_residues<N, CH>(chunk, dst, (int64_t)rows * pitch);
    }
}

// Row scales of a matrix stored column by column, src[(k0 + k) ld + r]: RB rows per block
// (consecutive lanes), the columns over its 1024 / RB groups of lanes.
template <int RB>
static __global__ void __launch_bounds__(1024)
row_scale_cols_kernel(const double *__restrict__ X, int64_t ld, int rows, int64_t K, float bits,
                      int *__restrict__ sc)
{
    constexpr int NG = 1024 / RB;
    __shared__ float sm[NG][RB + 1], sq[NG][RB + 1];
    __shared__ unsigned long long sb[NG][RB + 1];
    const int t = threadIdx.x % RB, g = threadIdx.x / RB;
    const int r = blockIdx.x * RB + t;
    // sums over the groups in a fixed order, left in a[0]
    auto reduce = [&](auto &a, auto op) {
        for (int h = NG / 2; h > 0; h >>= 1) {
            __syncthreads();
            if (g < h)
                a[g][t] = op(a[g][t], a[g + h][t]);
        }
        __syncthreads();
    };
    auto add = [](auto x, auto y) { return x + y; };
    auto larger = [](auto x, auto y) { return x > y ? x : y; };
    float m = 0.0f, ss = 0.0f;
    unsigned long long mb = 0;
    if (r < rows) {
#pragma unroll 4
        for (int64_t k = g; k < K; k += NG) {
            const double x = X[k * ld + r];
            const float v = abs_up(x);
            const unsigned long long b = abs_bits(x);
            m = fmaxf(m, v);
            ss = fmaf(v, v, ss);
            mb = b > mb ? b : mb;
        }
    }
    sm[g][t] = m;
    sq[g][t] = ss;
    sb[g][t] = mb;
    reduce(sm, larger);
    reduce(sq, add);
    reduce(sb, larger);
    int s = 0;
    const bool fast = scale_fast(sm[0][t], sq[0][t], bits, K, &s);
    if (__syncthreads_or(r < rows && !fast)) {
        mb = sb[0][t];
        const int e = max_exponent(mb);
        float s1 = 0.0f;
        double s2 = 0.0;
        if (r < rows && !fast)
            for (int64_t k = g; k < K; k += NG) {
                const float v = scaled_up(X[k * ld + r], e);
                if (K <= kFloatSums)
                    s1 = fmaf(v, v, s1);
                else
                    s2 += (double)v * v;
            }
        __syncthreads();  // sb[0] and sq[0] are read
        double(*sd)[RB + 1] = reinterpret_cast<double(*)[RB + 1]>(sb);
        sq[g][t] = s1;
        sd[g][t] = s2;
        if (K <= kFloatSums)
            reduce(sq, add);
        else
            reduce(sd, add);
        if (!fast)
            s = scale_slow(mb, K <= kFloatSums ? sq[0][t] : (float)sd[0][t], bits);
    }
    if (g != 0 || r >= rows)
        return;
    sc[r] = s;
}

// The residues of such a matrix, as residue_rows_kernel: 32 rows x 64 columns per block
// through shared memory (groups of eight columns four doubles further, so that eight
// lanes reading eight columns apart take the minimum two wavefronts), so that reads run
// along the rows and stores along the columns.
template <int N, bool kMag>
__global__ void __launch_bounds__(256)
residue_cols_kernel(const double *__restrict__ X, int64_t ld, int rows, int64_t k0, int64_t kp,
                    int64_t pitch, const int *__restrict__ sc, __nv_bfloat16 *__restrict__ planes)
{
    constexpr int CH = moduli::chunks(N);
    __shared__ double tile[64 * 32 + 8 * 4];
    const int64_t kb = (int64_t)blockIdx.x * 64;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row = threadIdx.x >> 3, kg = threadIdx.x & 7;
    for (int r0 = blockIdx.y * 32; r0 < rows; r0 += gridDim.y * 32) {
        __syncthreads();
        for (int k = warp; k < 64; k += 8)
            tile[k * 32 + (k >> 3) * 4 + lane] =
                (r0 + lane < rows && kb + k < kp) ? X[(k0 + kb + k) * ld + r0 + lane] : 0.0;
        __syncthreads();
        if (r0 + row >= rows || kb + kg * 8 >= pitch)
            continue;
        const int s = max(sc[r0 + row], -4096);
        double x[8];
        float v[8][CH];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            x[q] = tile[(kg * 8 + q) * 32 + kg * 4 + row];
            int_chunks<CH>(x[q], s, v[q]);
        }
        __nv_bfloat16 *dst = planes + (int64_t)(r0 + row) * pitch + kb + kg * 8;
        if constexpr (kMag)
            store_magnitudes(x, s, dst + N * (int64_t)rows * pitch);
        uint64_t chunk[CH][4];
        pack_chunks<N>(v, chunk);
        store_residues<N, CH>(chunk, dst, (int64_t)rows * pitch);
    }
}

// Scales and residues of short rows in one launch: G lanes per row, eight consecutive k per
// lane and step; a row of one step (K <= 8 G) is read once.  (A block per row for the scales
// and another for the residues leave most of their threads without work: 600 900 rows of
// 100 took 0.36 + 0.60 ms.)
template <int N, bool kMag, int G, class Src>
__global__ void __launch_bounds__(128)
residue_short_kernel(Src src, int r0, int rows, int K, int pitch, float bits,
                     int *__restrict__ sc, __nv_bfloat16 *__restrict__ planes)
{
    constexpr int CH = moduli::chunks(N);
    constexpr int kRows = 128 / G;  // rows per block
    using Value = typename ValueOf<Src::kDoubleFloat>::T;
    const int gl = threadIdx.x % G;
    const int64_t steps = ((int64_t)rows + kRows - 1) / kRows;
    for (int64_t b = blockIdx.x; b < steps; b += gridDim.x) {
        const int64_t r = b * kRows + threadIdx.x / G;
        const bool ok = r < rows;  // (every lane takes part in the reductions)
        Value x[8];
        auto load = [&](int kk) {
#pragma unroll
            for (int q = 0; q < 8; q++)
                x[q] = ok && kk + q < K ? value_of(src, r0 + r, kk + q) : Value{};
        };
        float m = 0.0f, ss = 0.0f;
        for (int kk = gl * 8; kk < K; kk += 8 * G) {
            load(kk);
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const float v = up_of(x[q]);
                m = fmaxf(m, v);
                ss = fmaf(v, v, ss);
            }
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
        }
        int s = 0;
        const bool fast = scale_fast(m, ss, bits, K, &s);
        if (!__all_sync(0xffffffffu, fast)) {
            unsigned long long mb = 0;
            if (ok)
                for (int k = gl; k < K; k += G) {
                    const unsigned long long v = abs_bits(src(r0 + r, k));
                    mb = v > mb ? v : mb;
                }
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1) {
                const unsigned long long v = __shfl_xor_sync(0xffffffffu, mb, o);
                mb = v > mb ? v : mb;
            }
            const int e = max_exponent(mb);
            float s2 = 0.0f;
            if (ok)
                for (int kk = gl * 8; kk < K; kk += 8 * G)  // (the order above)
                    for (int k = kk; k < min(K, kk + 8); k++) {
                        const float v = scaled_up(src(r0 + r, k), e);
                        s2 = fmaf(v, v, s2);
                    }
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1)
                s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            if (!fast)
                s = scale_slow(mb, s2, bits);
        }
        if (!ok)
            continue;
        if (gl == 0)
            sc[r0 + r] = s;
        s = max(s, -4096);
        const bool again = K > 8 * G;
        for (int kk = gl * 8; kk < pitch; kk += 8 * G) {
            if (again || kk >= K)
                load(kk);
            float v[8][CH];
#pragma unroll
            for (int q = 0; q < 8; q++)
                residue_chunks<N>(x[q], s, v[q]);
            if constexpr (kMag)
                store_magnitudes(x, s, planes + r * pitch + kk + N * (int64_t)rows * pitch);
            uint64_t chunk[CH][4];
            pack_chunks<N>(v, chunk);
            store_residues<N, CH>(chunk, planes + r * pitch + kk, (int64_t)rows * pitch);
        }
    }
}

// Host side.  Rows up to kShortRow long and in one panel take their scales with their
// residues (residue_rows, one launch fewer); others beforehand (row_scales).
constexpr int64_t kShortRow = 1024;

template <class Src>
static int row_scales(cudaStream_t st, Src src, int rows, int64_t K, int64_t k_panel, int n_mod,
                      int *sc)
{
    if (rows <= 0 || (K <= kShortRow && k_panel >= K))
        return CUTC_OK;
    row_scale_kernel<Src><<<std::min(rows, 1 << 20), 256, 0, st>>>(src, rows, K,
                                                                    moduli::row_bits(n_mod), sc);
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    return CUTC_OK;
}

// The planes of the K panel [k0, k0 + kp) for rows r0 .. r0 + rows; sc holds the scales of
// all rows (row_scales) or receives them.
template <int N, bool kMag = false, class Src>
static int residue_rows(cudaStream_t st, Src src, int r0, int rows, int64_t K, int64_t k0,
                        int64_t kp, int64_t pitch, int *sc, void *planes)
{
    if (rows <= 0 || kp <= 0)
        return CUTC_OK;
    auto *out = (__nv_bfloat16 *)planes;
    if (K <= kShortRow && kp == K) {
        auto launch = [&](auto g) {
            constexpr int G = decltype(g)::value;
            residue_short_kernel<N, kMag, G, Src><<<std::min(ceil_div(rows, 128 / G), 1u << 16), 128, 0, st>>>(
                src, r0, rows, (int)K, (int)pitch, moduli::row_bits(N), sc, out);
        };
        if (K <= 64)
            launch(std::integral_constant<int, 8>{});
        else if (K <= 128)
            launch(std::integral_constant<int, 16>{});
        else
            launch(std::integral_constant<int, 32>{});
    } else {
        dim3 grid(ceil_div(pitch, 8 * 128), (unsigned)std::min(rows, 65535));
        residue_rows_kernel<N, kMag, Src><<<grid, 128, 0, st>>>(src, r0, rows, k0, kp, pitch, sc, out);
    }
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    return CUTC_OK;
}

template <class Src>
static int residue_rows(cudaStream_t st, int n_mod, Src src, int r0, int rows, int64_t K,
                        int64_t k0, int64_t kp, int64_t pitch, int *sc, void *planes)
{
    switch (n_mod) {
    case 8: return residue_rows<8>(st, src, r0, rows, K, k0, kp, pitch, sc, planes);
    case 9: return residue_rows<9>(st, src, r0, rows, K, k0, kp, pitch, sc, planes);
    case 10: return residue_rows<10>(st, src, r0, rows, K, k0, kp, pitch, sc, planes);
    case 11: return residue_rows<11>(st, src, r0, rows, K, k0, kp, pitch, sc, planes);
    case 12: return residue_rows<12>(st, src, r0, rows, K, k0, kp, pitch, sc, planes);
    case 13: return residue_rows<13>(st, src, r0, rows, K, k0, kp, pitch, sc, planes);
    case 15: return residue_rows<15>(st, src, r0, rows, K, k0, kp, pitch, sc, planes);
    case 17: return residue_rows<17>(st, src, r0, rows, K, k0, kp, pitch, sc, planes);
    }
    cutc_set_error(CUTC_ERR_INVALID, "no residue kernel for %d moduli", n_mod);
    return CUTC_ERR_INVALID;
}

static inline int row_scales_cols(cudaStream_t st, const double *X, int64_t ld, int rows,
                                  int64_t K, int n_mod, int *sc)
{
    if (rows <= 0)
        return CUTC_OK;
    // few rows: 64-byte runs and four times the blocks (300 rows of 9000: 100 us with 32 rows
    // a block)
    const float bits = moduli::row_bits(n_mod);
    if (rows <= 32 * device_sms())
        row_scale_cols_kernel<8><<<ceil_div(rows, 8), 1024, 0, st>>>(X, ld, rows, K, bits, sc);
    else
        row_scale_cols_kernel<32><<<ceil_div(rows, 32), 1024, 0, st>>>(X, ld, rows, K, bits, sc);
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    return CUTC_OK;
}

template <int N, bool kMag = false>
static int residue_cols(cudaStream_t st, const double *X, int64_t ld, int rows, int64_t k0,
                        int64_t kp, int64_t pitch, const int *sc, void *planes)
{
    if (rows <= 0 || kp <= 0)
        return CUTC_OK;
    dim3 grid(ceil_div(pitch, 64), std::min(ceil_div(rows, 32), 65535u));
    residue_cols_kernel<N, kMag><<<grid, 256, 0, st>>>(X, ld, rows, k0, kp, pitch, sc,
                                                 (__nv_bfloat16 *)planes);
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    return CUTC_OK;
}

static inline int residue_cols(cudaStream_t st, int n_mod, const double *X, int64_t ld, int rows,
                               int64_t k0, int64_t kp, int64_t pitch, const int *sc, void *planes)
{
    switch (n_mod) {
    case 8: return residue_cols<8>(st, X, ld, rows, k0, kp, pitch, sc, planes);
    case 9: return residue_cols<9>(st, X, ld, rows, k0, kp, pitch, sc, planes);
    case 10: return residue_cols<10>(st, X, ld, rows, k0, kp, pitch, sc, planes);
    case 11: return residue_cols<11>(st, X, ld, rows, k0, kp, pitch, sc, planes);
    case 12: return residue_cols<12>(st, X, ld, rows, k0, kp, pitch, sc, planes);
    case 13: return residue_cols<13>(st, X, ld, rows, k0, kp, pitch, sc, planes);
    case 15: return residue_cols<15>(st, X, ld, rows, k0, kp, pitch, sc, planes);
    case 17: return residue_cols<17>(st, X, ld, rows, k0, kp, pitch, sc, planes);
    }
    cutc_set_error(CUTC_ERR_INVALID, "no residue kernel for %d moduli", n_mod);
    return CUTC_ERR_INVALID;
}

}  // namespace cutc
