// Pair terms grad1 u(r1, r2) on the tensor cores (tcgen05 + TMA).
//
// For fixed g12 the nucleus sum of grad1 u(r1, r2) is the contraction
//   V_c(r1, r2) = sum_k C[(r1, c)][k] F[r2][k],  k over (nucleus, power of f2)
// (pair_df.cu builds F and the coefficient rows C per r1 point in FP64), and the pair's
// value a polynomial in g12 of the V_c: 16 rows and four powers per nucleus where every
// Jastrow exponent is 0, 2, 3 or 4, 32 rows and seven powers for any exponents up to 6.
// The contraction runs on operands split into S slices,
//     A[r, k] = 2^{e_r} sum_{s < S} a_s[r, k],  a_s = q_s 2^{-8-9s},  q_s in [-256, 256]
// (S signed 9-bit digits of the row-scaled value), whose products a_s b_t, s + t < S, run
// as BF16 tcgen05.mma with one FP32 accumulator per diagonal d = s + t: the S slices of b
// are stacked in shared memory, so one instruction per slice of a takes all of them (the
// error-free splitting of Ozaki, Ogita, Oishi and Rump 2012).  A product of diagonal d is
// a multiple of 2^{-16-9d}, at most 2^{-9d}, so the FP32 sums are exact while
// (d + 1) K 2^16 <= 2^24: K <= 85 for d <= 2 (double-float results), K <= 64 for d <= 3
// (FP64 results); later diagonals round at 2^-27 2^-24 and 2^-36 2^-24 of the row scales.
// With more nuclei K is cut into groups of 64, one launch each, whose V values are added
// (FP64: as integers) through device memory: 16 to 384 bytes a pair and group, a few
// percent of what the kernels that loop over the nuclei take.
//
// A = the F slices of 128 r2 points, all of K, loaded once per CTA; B = the coefficient
// slices in tiles of 64 rows (four r1 points, or two; one point for FP64 results), streamed
// (whole tiles, or K block by K block where three checked blocks would not fit);
// one stacked accumulator set in tensor memory (four or two for FP64 results).  The tensor-core work of a tile is a small part of its epilogue, so
// one B stage per accumulator set suffices: the next tile's MMAs run as soon as the
// epilogue has read the accumulators, and one control warp issues both the TMA loads and
// the MMAs.
//
// Double-float epilogue (lane = r2 point, one r1 point per warp): the S diagonals of the
// point's columns are added exactly on fixed grids into double-float values, then g12 and
// its gradient, the polynomial, -1/2 |grad u|^2 and the (hi, lo) G planes follow in
// double-float, with FP64 coordinate differences near e-e coalescence.  About 800 FP32
// operations per pair with 16 rows instead of 30 df multiply-adds (~450 operations) per
// nucleus.
//
// F and the coefficients enter with an error relative to their rows' maxima, where a term by
// term sum's is relative to the terms.  So FP64 results, and those in double-float of general
// exponents and of more than 20 nuclei (from 6 slices), are checked: one more product, of the
// operands' magnitudes to 8 bits (plane S, accumulators of its own), gives
// v_c = sum_k |C[(r1, c)][k]| F[r2][k], and with it the sums of the terms' magnitudes and of the
// errors, both as polynomials in g12.  The error of V_c is about sqrt(K) 2^-63 of the row
// scales with seven slices (rms, from the slices and the products left out), sqrt(K) 2^-54 with
// six; pairs for which four times that is above 2^-53 (2^-45) of the terms (r2 near a nucleus whose terms all vanish there, small
// values of few nuclei: fewer than one in 10^4 of 8 nuclei with 13 terms) are marked in a bit
// mask and formed again term by term behind the kernel (pair.cu).
//
// FP64 epilogue: the diagonals down to 2^-43 of the row scales become one exact integer
// and a double in integer arithmetic, the rest stays in FP32 beside it, and g12, its
// gradient and the polynomial take FP64: 45 FP64 operations per pair with 16 rows, whatever
// the number of nuclei, on a pipe of 2 per clock and SM, against about 11 per term in the
// term-by-term kernel (pair.cu).  512 x 20 011 pairs, 8 nuclei with 13
// terms each: 19.4 -> 1.22 ms.  General exponents in double-float, 2003 x 30 011 pairs, 6
// nuclei, against pair_df_kernel<6>: 16.6 -> 5.1 ms.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>

#include "common.cuh"
#include "dfloat.cuh"
#include "digits.cuh"
#include "modular.cuh"
#include "pair_tc.cuh"
#include "series.cuh"
#include "tc.cuh"

namespace cutc {

constexpr int kBM = 128;        // r2 points per CTA (TMEM lanes)
constexpr int kBK = 32;         // K per TMA box: 32 BF16 = 64-byte rows (64B swizzle)
constexpr uint32_t kTmemCols = 512;
constexpr int kPairBN = 64;     // coefficient rows per N tile
constexpr int kNanExponent = 1025;  // row exponent of a row with an infinity or a NaN

struct PairTcParams {
    int tiles_m, tiles_n, chunk;  // r2 tiles of 128 points, N tiles, N tiles per CTA
    int Mpad, Npad;               // padded rows of the F and coefficient slices
    const int *ea, *eb;           // row exponents of the F and the coefficient slices
    const float *bscale;          // 2^(row exponent) of each coefficient row, 0 for a zero row
    const float2 *r1d;            // double-float: the tile's r1 points, [3 i + c]
    PairDfArgs P;                 // geometry and outputs
    double *G64;                  // FP64: in place of P.G
    float check;                  // checked: 2^8 / sqrt(K), double-float 2^7 / sqrt(K)
    unsigned *marks;              // checked: bit j % 32 of marks[i mark_words + j / 32]: (i, j) is
    int mark_words;               // left out, and *marked is set
    int *marked;
    int *err;
    // a group of K blocks of a longer contraction: from block kb0 on; the values so far are
    // added (not for the first group), and kept (not for the last) at
    // part[(i R + c) n2 + j] (double-float), partI and partL (FP64: integer and rest)
    int kb0, first, last;
    float2 *part;
    long long *partI;
    float *partL, *partA;         // (and the magnitudes' sums)
};

// x 2^e for the scale of a value of row exponents e (clamped to the float range); NaN for
// a row that is not finite
__device__ __forceinline__ float pow2f(int e)
{
    if (e >= kNanExponent)
        return __int_as_float(0x7fffffff);
    e = e < -126 ? -126 : (e > 127 ? 127 : e);
    return __int_as_float((e + 127) << 23);
}

// R: coefficient rows per r1 point (16 or 32).
// CHK: with the magnitudes' product and the check (always with F64).
template <int S, int KB, int R, bool F64, bool CHK>
struct PairTcCfg {
    // Double-float: one accumulator set, and a warp per lane quarter and point of a tile
    // (16 warps with 16 rows, four per SM sub-partition, to hide the latency of their
    // dependent chains; 8 with 32 rows).  FP64: tiles of one point in four accumulator sets
    // (two with 32 rows), each with four warps of its own, so that one set's integer work
    // runs beside another's FP64 work (with one set, every warp waits for the same tile and
    // the FP64 pipe idled 40% of the time).
    static constexpr int kBN = F64 ? R : kPairBN;
    static constexpr int kBufs = F64 ? 64 / R : 1;
    static constexpr int kPts = kBN / R;
    static constexpr int kEpiWarps = F64 ? 4 * kBufs : 4 * kPts;
    static constexpr int kBufWarps = kEpiWarps / kBufs;  // epilogue warps of a buffer
    static constexpr int kCtlWarp = kEpiWarps;       // TMA loads and MMAs, lane 0
    static constexpr int kThreads = (kEpiWarps + 1) * 32;
    static constexpr int kPlanes = S + (CHK ? 1 : 0);  // slices, and the magnitudes
    static constexpr int kASlice = kBM * kBK * 2;
    static constexpr int kBSlice = kBN * kBK * 2;
    static constexpr int kABytes = KB * kPlanes * kASlice;
    // B comes in units: all of a tile's K with a stage per accumulator set, or one K block
    // with two stages where the planes of three blocks do not fit
    static constexpr bool kSplit = CHK && KB == 3;
    static constexpr int kUnits = kSplit ? KB : 1;   // per tile
    static constexpr int kUnitBlocks = KB / kUnits;
    static constexpr int kStages = kSplit ? 2 : kBufs;
    static constexpr int kBStage = kUnitBlocks * kPlanes * kBSlice;
    static constexpr int kBufCols = kBN * kPlanes;   // accumulator columns of a buffer
    static constexpr int kSmem = kABytes + kStages * kBStage + 1024 + 256;
    static constexpr int kMaxN = 256;                // widest kind::f16 instruction at M = 128
    static_assert(kSmem <= 227 * 1024, "shared memory");
    static_assert(kBufs * kBufCols <= (int)kTmemCols, "accumulators exceed tensor memory");
    static_assert(kMaxN % kBN == 0, "instruction splits on diagonal boundaries");
    static_assert(kBSlice % 512 == 0, "B slices must stack on 8-row swizzle atoms");
};

// The V values of R columns of the warp's lanes, in double-float: the diagonals summed
// exactly on grids.  In units of the row scales every diagonal sum D_d is a multiple of
// 2^(-16-9d) and |D_0| <= K:
//   H  = D_0 + D_1 rounded to multiples of 2^-16      (exact: below 2^7 there)
//   L  = the rest of D_1 + D_2 rounded to 2^-25         (exact: below 2^-8 there)
//   L2 = the rest of D_2 + D_3 + ... (FP32; below 2^-18, so off by < 2^-42)
// Two columns share each packed f32x2 operation.
template <int S>
__device__ __forceinline__ void read_df16(uint32_t cb, uint64_t (&H)[8], uint64_t (&L)[8],
                                          uint64_t (&L2)[8])
{
    const uint64_t C16 = tc::f2_dup(192.0f), C25 = tc::f2_dup(0.375f);
    float v[16];
    tc::tmem_ld16(cb, v);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        H[k] = tc::f2_pack(__float_as_uint(v[2 * k]), __float_as_uint(v[2 * k + 1]));
        L[k] = L2[k] = 0ull;
    }
#pragma unroll
    for (int d = 1; d < S; d++) {
        tc::tmem_ld16(cb + (uint32_t)(kPairBN * d), v);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint64_t x = tc::f2_pack(__float_as_uint(v[2 * k]), __float_as_uint(v[2 * k + 1]));
            if (d == 1) {
                const uint64_t hh = tc::f2_sub(tc::f2_add(x, C16), C16);
                H[k] = tc::f2_add(H[k], hh);
                L[k] = tc::f2_sub(x, hh);
            } else if (d == 2) {
                const uint64_t hh = tc::f2_sub(tc::f2_add(x, C25), C25);
                L[k] = tc::f2_add(L[k], hh);
                L2[k] = tc::f2_sub(x, hh);
            } else {
                L2[k] = tc::f2_add(L2[k], x);
            }
        }
    }
}

// V_c 2^-ea = 2^eb_c ((H + L) + L2): TwoSum of H and L, then the rest.  The F rows' scale
// 2^ea, a power of two common to a pair's values, multiplies the results instead (the
// polynomial is linear in V, and power-of-two scaling commutes with double-float
// arithmetic).
__device__ __forceinline__ void scale_df16(const uint64_t (&H)[8], const uint64_t (&L)[8],
                                           const uint64_t (&L2)[8], const float *scr, df::D *V)
{
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const uint64_t sm = tc::f2_add(H[k], L[k]);
        const uint64_t bb = tc::f2_sub(sm, H[k]);
        uint64_t e = tc::f2_add(tc::f2_sub(H[k], tc::f2_sub(sm, bb)), tc::f2_sub(L[k], bb));
        e = tc::f2_add(e, L2[k]);
        const uint64_t sc = *reinterpret_cast<const uint64_t *>(scr + 2 * k);
        const uint64_t hs = tc::f2_mul(sm, sc), ls = tc::f2_mul(e, sc);
        V[2 * k] = df::make(tc::f2_lo(hs), tc::f2_lo(ls));
        V[2 * k + 1] = df::make(tc::f2_hi(hs), tc::f2_hi(ls));
    }
}

// Whether the error of a pair's values may be above that of a term by term sum (the check at
// the top of this file): w[c] = 2^eb_c (check v_c - 1), the margin of V_c.
template <int R>
__device__ __forceinline__ bool pair_unsure(const float *w, float g, float gx, float gy, float gz)
{
    float ux, uy, uz, dudg;
    if constexpr (R == 16) {
        const float g2 = g * g;
        auto poly = [&](int c) { return fmaf(fmaf(fmaf(w[c + 3], g, w[c + 2]), g, w[c + 1]), g2, w[c]); };
        ux = poly(0);
        uy = poly(4);
        uz = poly(8);
        dudg = fmaf(fmaf(w[14], g, w[13]), g, w[12]) * g;
    } else {
        auto poly = [&](int c, int n) {
            float s = w[c + n - 1];
#pragma unroll
            for (int o = n - 2; o >= 0; o--)
                s = fmaf(s, g, w[c + o]);
            return s;
        };
        ux = poly(0, 7);
        uy = poly(7, 7);
        uz = poly(14, 7);
        dudg = poly(21, 6);
    }
    // (a NaN is unsure)
    return !(fmaf(dudg, fabsf(gx), ux) >= 0.f && fmaf(dudg, fabsf(gy), uy) >= 0.f &&
             fmaf(dudg, fabsf(gz), uz) >= 0.f);
}

// One pair in double-float from its V values; with CHK true, and nothing is written, when they
// are unsure.
template <int R, bool CHK>
__device__ __forceinline__ bool pair_df(const PairTcParams &Q, int i, int j, const df::D *V,
                                        const float *w, float2 x2, float2 y2, float2 z2, float sa,
                                        df::D a)
{
    const PairDfArgs &P = Q.P;
    const float2 *r1p = Q.r1d + 3 * (int64_t)i;
    const float2 r1x = r1p[0], r1y = r1p[1], r1z = r1p[2];
    df::D dx = df::sub(df::make(r1x.x, r1x.y), df::make(x2.x, x2.y));
    df::D dy = df::sub(df::make(r1y.x, r1y.y), df::make(y2.x, y2.y));
    df::D dz = df::sub(df::make(r1z.x, r1z.y), df::make(z2.x, z2.y));
    df::D d2 = df::add(df::add(df::sqr(dx), df::sqr(dy)), df::sqr(dz));
    bool coalesced = false;
    if (d2.hi < kNearPairR2) {
        // near e-e coalescence the differences are taken in FP64, where they are
        // exact (the coordinates' double-float forms keep only 48 bits); only g12
        // and its gradient depend on them, so the rest stays as it is.  The
        // reference's own guard, r12^2 <= 1e-15 (src/jast_bh.cu:143), gives g = 0.
        const double *a1 = P.r1 + 3 * (int64_t)(P.i0 + i);
        const double *a2 = P.r2 + 3 * (int64_t)j;
        const double ex = a1[0] - a2[0], ey = a1[1] - a2[1], ez = a1[2] - a2[2];
        dx = df::from_double(ex);
        dy = df::from_double(ey);
        dz = df::from_double(ez);
        d2 = df::add(df::add(df::sqr(dx), df::sqr(dy)), df::sqr(dz));
        coalesced = !(ex * ex + ey * ey + ez * ez > 1e-15);
    }
    df::D g = {0.f, 0.f}, gx = {0.f, 0.f}, gy = {0.f, 0.f}, gz = {0.f, 0.f};
    if (!coalesced) {
        const df::D rd = df::sqrt(d2);
        const df::D ar = df::mul(rd, a);
        const df::D t = df::recip(df::add_f(ar, 1.0f));
        g = df::mul(ar, t);
        const df::D sg = df::mul(df::mul(df::sqr(t), a), df::recip(rd));
        gx = df::mul(sg, dx);
        gy = df::mul(sg, dy);
        gz = df::mul(sg, dz);
    }
    if constexpr (CHK)
        if (pair_unsure<R>(w, g.hi, gx.hi, gy.hi, gz.hi))
            return true;
    df::D ux, uy, uz, dudg;
    if constexpr (R == 16) {
        const df::D g2 = df::sqr(g);
        // sum_o g^o V_o, o = 0, 2, 3, 4
        ux = df::fma(df::fma(df::fma(V[3], g, V[2]), g, V[1]), g2, V[0]);
        uy = df::fma(df::fma(df::fma(V[7], g, V[6]), g, V[5]), g2, V[4]);
        uz = df::fma(df::fma(df::fma(V[11], g, V[10]), g, V[9]), g2, V[8]);
        dudg = df::mul(df::fma(df::fma(V[14], g, V[13]), g, V[12]), g);
    } else {
        auto horner = [&](const df::D *v, int n) {
            df::D s = v[n - 1];
#pragma unroll
            for (int o = n - 2; o >= 0; o--)
                s = df::fma(s, g, v[o]);
            return s;
        };
        ux = horner(V, 7);
        uy = horner(V + 7, 7);
        uz = horner(V + 14, 7);
        dudg = horner(V + 21, 6);
    }
    ux = df::fma(dudg, gx, ux);
    uy = df::fma(dudg, gy, uy);
    uz = df::fma(dudg, gz, uz);
    ux = df::make(__fmul_rn(ux.hi, sa), __fmul_rn(ux.lo, sa));
    uy = df::make(__fmul_rn(uy.hi, sa), __fmul_rn(uy.lo, sa));
    uz = df::make(__fmul_rn(uz.hi, sa), __fmul_rn(uz.lo, sa));
    const df::D n2v = df::add(df::add(df::sqr(ux), df::sqr(uy)), df::sqr(uz));
    const df::D lv = df::mul_f(n2v, -0.5f);
    float2 *o = P.G + (int64_t)i * P.ldg + j;
    o[0] = make_float2(ux.hi, ux.lo);
    o[P.plane] = make_float2(uy.hi, uy.lo);
    o[2 * P.plane] = make_float2(uz.hi, uz.lo);
    o[3 * P.plane] = make_float2(lv.hi, lv.lo);
    return false;
}

// I 2^k for |I| < 2^53, exactly, in integer arithmetic (0 below the normal range, an
// infinity above it).  A V value is at most K units of the row scales, K 2^43 as an integer, and
// K at most 7 powers of kMaxNuc nuclei in all groups together.
static_assert(7 * kMaxNuc < 1024, "the V values' integers");
__device__ __forceinline__ double int_double(long long I, int k)
{
    const unsigned long long m = (unsigned long long)(I < 0 ? -I : I);
    const int lz = __clzll((long long)m);  // 64 for 0
    const int E = 1023 + 63 - lz + k;      // the exponent field
    const unsigned long long f = m << ((lz - 11) & 63);  // leading bit at 52
    unsigned hi = (unsigned)(f >> 32) + ((unsigned)(E - 1) << 20), lo = (unsigned)f;
    if (m == 0 || E < 1)
        hi = lo = 0u;
    else if (E > 2046) {
        hi = 0x7ff00000u;
        lo = 0u;
    }
    return __hiloint2double((int)(hi | ((unsigned)(I >> 32) & 0x80000000u)), (int)lo);
}

// The V values of eight columns, in units of the row scales, in two parts each: an integer
// multiple of 2^-43 and the rest (below 2^-35, to 2^-60) as a float:
//   H + L + L2 + L3 on the grids 2^-16, 2^-25, 2^-34, 2^-43 (each exact, as read_df16)
// is the integer, below 2^50, formed with integer operations.
template <int S, int BN>
__device__ __forceinline__ void read_f64_8(uint32_t cb, long long *I, float *rest)
{
    static_assert(S == 7, "FP64 results take 7 slices");
    float v[8];
    uint64_t H[4], L[4], L2[4], L3[4], L4[4];
    tc::tmem_ld8(cb, v);
#pragma unroll
    for (int k = 0; k < 4; k++)
        H[k] = tc::f2_pack(__float_as_uint(v[2 * k]), __float_as_uint(v[2 * k + 1]));
    // multiples of 2^g: C = 1.5 2^(23 + g)
    auto cut = [&](int d, float C, uint64_t (&up)[4], uint64_t (&down)[4]) {
        const uint64_t Cg = tc::f2_dup(C);
        tc::tmem_ld8(cb + (uint32_t)(BN * d), v);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint64_t x = tc::f2_pack(__float_as_uint(v[2 * k]), __float_as_uint(v[2 * k + 1]));
            const uint64_t hh = tc::f2_sub(tc::f2_add(x, Cg), Cg);
            up[k] = tc::f2_add(up[k], hh);
            down[k] = tc::f2_sub(x, hh);
        }
    };
    cut(1, 192.0f, H, L);
    cut(2, 0.375f, L, L2);
    cut(3, 0.375f * 0x1p-9f, L2, L3);
    cut(4, 0.375f * 0x1p-18f, L3, L4);
#pragma unroll
    for (int d = 5; d < S; d++) {
        tc::tmem_ld8(cb + (uint32_t)(BN * d), v);
#pragma unroll
        for (int k = 0; k < 4; k++)
            L4[k] = tc::f2_add(L4[k], tc::f2_pack(__float_as_uint(v[2 * k]),
                                                  __float_as_uint(v[2 * k + 1])));
    }
    auto grid_int = [](float x, float s) {  // x s, an integer below 2^22
        return __float_as_int(__fmaf_rn(x, s, 12582912.0f)) - 0x4b400000;
    };
#pragma unroll
    for (int k = 0; k < 8; k++) {
        auto part = [&](const uint64_t (&p)[4]) { return k & 1 ? tc::f2_hi(p[k / 2]) : tc::f2_lo(p[k / 2]); };
        const int ih = __float2int_rn(part(H) * 65536.0f);
        const int il = grid_int(part(L), 0x1p25f);
        const int il2 = grid_int(part(L2), 0x1p34f), il3 = grid_int(part(L3), 0x1p43f);
        I[k] = ((long long)ih << 27) + ((long long)il << 18) + (long long)(il2 * 512 + il3);
        rest[k] = part(L4);
    }
}

// Their values: hi as a double (made in integer arithmetic: an FP64 add per value instead,
// on the pipe that bounds the kernel, cost 15 of 67 FP64 operations a pair) and lo as a
// float.  eb: the exponents of the columns' scales, ea: the F row's.
__device__ __forceinline__ void scale_f64(long long I, float rest, int eb, int ea, double *hi, float *lo)
{
    const int e = eb + ea;
    *hi = eb >= kNanExponent || ea >= kNanExponent ? __longlong_as_double(0x7ff8000000000000ll)
                                                   : int_double(I, e - 43);
    *lo = rest * pow2f(min(e, 127));
}

// any float as a double (subnormals as zero, infinities and NaNs as infinities or NaNs)
__device__ __forceinline__ double signed_double(float x)
{
    const unsigned b = __float_as_uint(x), m = b & 0x7fffffffu;
    unsigned hi = (m >> 3) + 0x38000000u;
    hi = m < 0x00800000u ? 0u : m >= 0x7f800000u ? (m >> 3) | 0x7ff00000u : hi;
    return __hiloint2double((int)(hi | (b & 0x80000000u)), m < 0x00800000u ? 0 : (int)(m << 29));
}

// -x / 2 of a finite normal x, else by an FP64 multiply
__device__ __forceinline__ double minus_half(double x)
{
    const int hi = __double2hiint(x);
    const int E = (hi >> 20) & 0x7ff;
    if (E >= 2 && E < 0x7ff)
        return __hiloint2double((hi - 0x00100000) ^ (int)0x80000000, __double2loint(x));
    return -0.5 * x;
}

// One pair in FP64 from its V values (hi + lo); true, and nothing is written, when they are
// unsure.
template <int R>
__device__ __forceinline__ bool pair_f64(const PairTcParams &Q, int i, int j, const double *V,
                                         const float *W, const float *w, double x2, double y2,
                                         double z2)
{
    const PairDfArgs &P = Q.P;
    const double *r1p = P.r1 + 3 * (int64_t)(P.i0 + i);
    const double a = P.a_ee;
    const bool a_one = __double_as_longlong(a) == 0x3ff0000000000000ll;  // the reference's scale
    const double dx = r1p[0] - x2, dy = r1p[1] - y2, dz = r1p[2] - z2;
    const double d2 = fma(dx, dx, fma(dy, dy, dz * dz));
    const int hw = __double2hiint(d2);
    double g = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
    // d2 > 1e-15 (src/jast_bh.cu:143) on the bits: positive doubles order like them, and a
    // NaN is not greater
    const long long db = __double_as_longlong(d2);
    if (db > __double_as_longlong(1e-15) && db <= 0x7ff0000000000000ll) {
        double y, z, d;
        if (hw < (1023 + 120) << 20) {
            y = rsqrt_series(d2);
            d = d2 * y;
        } else {  // distances beyond 2^60, and infinities
            d = sqrt(d2);
            y = 1.0 / d;
        }
        const double ad = a_one ? d : a * d;
        const double den = 1.0 + ad;
        z = __double2hiint(den) < (1023 + 120) << 20 ? recip_series(den) : 1.0 / den;
        g = ad * z;
        double s = z * z * y;
        if (!a_one)
            s *= a;
        gx = s * dx;
        gy = s * dy;
        gz = s * dz;
    }
    const float gf = trunc_float(g);
    if (pair_unsure<R>(w, gf, trunc_float(gx), trunc_float(gy), trunc_float(gz)))
        return true;
    double ux, uy, uz, dudg;
    float lx, ly, lz, lg;
    if constexpr (R == 16) {
        const double g2 = g * g;
        const float gf2 = gf * gf;
        auto poly = [&](int c) { return fma(fma(fma(V[c + 3], g, V[c + 2]), g, V[c + 1]), g2, V[c]); };
        auto low = [&](int c) { return fmaf(fmaf(fmaf(W[c + 3], gf, W[c + 2]), gf, W[c + 1]), gf2, W[c]); };
        ux = poly(0);
        uy = poly(4);
        uz = poly(8);
        dudg = fma(fma(V[14], g, V[13]), g, V[12]) * g;
        lx = low(0);
        ly = low(4);
        lz = low(8);
        lg = fmaf(fmaf(W[14], gf, W[13]), gf, W[12]) * gf;
    } else {
        auto poly = [&](int c, int n) {
            double s = V[c + n - 1];
#pragma unroll
            for (int o = n - 2; o >= 0; o--)
                s = fma(s, g, V[c + o]);
            return s;
        };
        auto low = [&](int c, int n) {
            float s = W[c + n - 1];
#pragma unroll
            for (int o = n - 2; o >= 0; o--)
                s = fmaf(s, gf, W[c + o]);
            return s;
        };
        ux = poly(0, 7);
        uy = poly(7, 7);
        uz = poly(14, 7);
        dudg = poly(21, 6);
        lx = low(0, 7);
        ly = low(7, 7);
        lz = low(14, 7);
        lg = low(21, 6);
    }
    ux = fma(dudg, gx, ux) + signed_double(fmaf(lg, trunc_float(gx), lx));
    uy = fma(dudg, gy, uy) + signed_double(fmaf(lg, trunc_float(gy), ly));
    uz = fma(dudg, gz, uz) + signed_double(fmaf(lg, trunc_float(gz), lz));
    double *o = Q.G64 + (int64_t)i * P.ldg + j;
    o[0] = ux;
    o[P.plane] = uy;
    o[2 * P.plane] = uz;
    o[3 * P.plane] = minus_half(fma(ux, ux, fma(uy, uy, uz * uz)));
    return false;
}

// PART: one group of K blocks of a longer contraction (Q.kb0, Q.first, Q.last).
template <int S, int KB, int R, bool F64, bool CHK, bool PART>
__global__ void __launch_bounds__(PairTcCfg<S, KB, R, F64, CHK>::kThreads, 1)
pair_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ PairTcParams Q)
{
    using Cfg = PairTcCfg<S, KB, R, F64, CHK>;
    constexpr int D = S - 1, BN = Cfg::kBN, NP = Cfg::kPlanes;
    constexpr int kCtlWarp = Cfg::kCtlWarp;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem;
    uint8_t *sB = smem + Cfg::kABytes;
    constexpr int NB = Cfg::kBufs;
    constexpr int NS = Cfg::kStages, U = Cfg::kUnits;
    uint64_t *bars = reinterpret_cast<uint64_t *>(sB + NS * Cfg::kBStage);
    uint64_t *afull = bars;            // the F tile has landed
    uint64_t *full = bars + 1;         // a B stage holds a unit
    uint64_t *empty = full + NS;       // the MMAs of the unit are done with the B stage
    uint64_t *tfull = empty + NS;      // the accumulators hold the tile
    uint64_t *tempty = tfull + NB;     // its epilogue warps have read them
    uint64_t *drain = tempty + NB;
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(drain + 1);
    volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);

    const PairDfArgs &P = Q.P;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = (int)(blockIdx.x % Q.tiles_m) * kBM;
    const int t_begin = (int)(blockIdx.x / Q.tiles_m) * Q.chunk;
    const int ntiles = min(Q.tiles_n, t_begin + Q.chunk) - t_begin;

    if (threadIdx.x == 0) {
        tc::mbar_init(tc::smem_u32(afull), 1);
        for (int i = 0; i < NS; i++) {
            tc::mbar_init(tc::smem_u32(&full[i]), 1);
            tc::mbar_init(tc::smem_u32(&empty[i]), 1);
        }
        for (int i = 0; i < NB; i++) {
            tc::mbar_init(tc::smem_u32(&tfull[i]), 1);
            tc::mbar_init(tc::smem_u32(&tempty[i]), Cfg::kBufWarps);
        }
        tc::mbar_init(tc::smem_u32(drain), 1);
        *s_abort = 0;
        tc::fence_mbar_init();
    }
    if (warp == kCtlWarp) {
        tc::tmem_alloc(tc::smem_u32(s_tmem), kTmemCols);
        tc::tmem_relinquish();
        if (lane == 0) {
            tc::tma_prefetch(&tmA);
            tc::tma_prefetch(&tmB);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = *s_tmem;

    auto fail = [&](int code) {
        *s_abort = 1;
        atomicExch(Q.err, code);
    };

    if (warp == kCtlWarp) {
        if (lane == 0) {
            const int kb0 = PART ? Q.kb0 : 0;
            constexpr int UB = Cfg::kUnitBlocks;
            const int units = ntiles * U;
            auto load_b = [&](int u) {
                const int b = u % NS;
                const uint32_t fb = tc::smem_u32(&full[b]);
                tc::mbar_arrive_expect_tx(fb, Cfg::kBStage);
                const int n0 = (t_begin + u / U) * BN, k0 = kb0 + u % U * UB;
#pragma unroll
                for (int kb = 0; kb < UB; kb++)
#pragma unroll
                    for (int t = 0; t < NP; t++)
                        tc::tma_load_2d(
                            tc::smem_u32(sB + b * Cfg::kBStage + (kb * NP + t) * Cfg::kBSlice), &tmB,
                            (k0 + kb) * kBK, t * Q.Npad + n0, fb);
            };
            const uint32_t ab = tc::smem_u32(afull);
            tc::mbar_arrive_expect_tx(ab, Cfg::kABytes);
#pragma unroll
            for (int kb = 0; kb < KB; kb++)
#pragma unroll
                for (int s = 0; s < NP; s++)
                    tc::tma_load_2d(tc::smem_u32(sA + (kb * NP + s) * Cfg::kASlice), &tmA,
                                    (kb0 + kb) * kBK, s * Q.Mpad + m0, ab);
            int loaded = 0;  // B units issued
            for (; loaded < min(NS, units); loaded++)
                load_b(loaded);
            bool ok = tc::mbar_wait(ab, 0, s_abort);
            if (!ok)
                fail(12);
            for (int q = 0; q < ntiles && ok; q++) {
                const int set = q % NB, round = q / NB;
                // the accumulators are free once their epilogue warps have read the last tile
                if (round >= 1 &&
                    !tc::mbar_wait(tc::smem_u32(&tempty[set]), (round - 1) & 1, s_abort)) {
                    fail(13);
                    break;
                }
                const uint32_t acc = tbase + (uint32_t)(Cfg::kBufCols * set);
                bool first = true;
#pragma unroll
                for (int un = 0; un < U && ok; un++) {
                    const int u = q * U + un, b = u % NS;
                    if (!tc::mbar_wait(tc::smem_u32(&full[b]), (u / NS) & 1, s_abort)) {
                        fail(14);
                        ok = false;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint32_t sb0 = tc::smem_u32(sB + b * Cfg::kBStage);
                    const uint32_t sa0 = tc::smem_u32(sA) + un * UB * NP * Cfg::kASlice;
#pragma unroll
                    for (int kb = 0; kb < UB; kb++) {
#pragma unroll
                        for (int k16 = 0; k16 < kBK / 16; k16++) {
#pragma unroll
                            for (int s = 0; s < S; s++) {
                                // a_s x [b_0 .. b_{D-s}] -> diagonals s .. D, in instructions
                                // of at most kMaxN columns
                                const uint64_t ad = tc::smem_desc_sw64(
                                    sa0 + (kb * NP + s) * Cfg::kASlice + k16 * 32);
#pragma unroll
                                for (int t0 = 0; t0 <= D - s; t0 += Cfg::kMaxN / BN) {
                                    const int nt = min(Cfg::kMaxN / BN, D - s + 1 - t0);
                                    const uint64_t bd = tc::smem_desc_sw64(
                                        sb0 + (kb * NP + t0) * Cfg::kBSlice + k16 * 32);
                                    tc::mma_bf16(acc + (uint32_t)(BN * (s + t0)), ad, bd,
                                                 tc::idesc_bf16_f32(kBM, BN * nt), first ? 0u : 1u);
                                }
                                first = false;
                            }
                            if constexpr (CHK)  // the magnitudes' sums
                                tc::mma_bf16(
                                    acc + (uint32_t)(BN * S),
                                    tc::smem_desc_sw64(sa0 + (kb * NP + S) * Cfg::kASlice + k16 * 32),
                                    tc::smem_desc_sw64(sb0 + (kb * NP + S) * Cfg::kBSlice + k16 * 32),
                                    tc::idesc_bf16_f32(kBM, BN),
                                    un > 0 || kb > 0 || k16 > 0 ? 1u : 0u);
                        }
                    }
                    tc::mma_commit(tc::smem_u32(&empty[b]));
                    if (un == U - 1)
                        tc::mma_commit(tc::smem_u32(&tfull[set]));
                    // refill a B stage once its MMAs have read it: with several stages, that
                    // of the unit before, so that this wait does not hold up the next MMAs
                    const int r = NS > 1 ? u - 1 : u;
                    if (r >= 0 && loaded < units) {
                        if (!tc::mbar_wait(tc::smem_u32(&empty[r % NS]), (r / NS) & 1, s_abort)) {
                            fail(11);
                            ok = false;
                            break;
                        }
                        load_b(loaded++);
                    }
                }
            }
            tc::mma_commit(tc::smem_u32(drain));
            if (!tc::mbar_wait(tc::smem_u32(drain), 0, nullptr))
                fail(15);
            // let the copies still in flight land before the CTA goes away
            tc::mbar_wait(ab, 0, nullptr);
            if (*s_abort)
                for (int u = max(0, loaded - NS); u < loaded; u++)
                    tc::mbar_wait(tc::smem_u32(&full[u % NS]), (u / NS) & 1, nullptr);
        }
    } else {
        // ---- epilogue: the warp's r1 points of each N tile, 32 r2 points ----------------
        const int quarter = warp & 3, buf = NB == 1 ? 0 : warp >> 2;
        const int pt0 = NB == 1 ? warp >> 2 : 0;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        const int j = m0 + quarter * 32 + lane;
        const bool jok = j < P.n2;
        const int jc = jok ? j : 0;
        const int ea = Q.ea[jc];  // F rows: 1 where the row maximum is f^0 = 1
        float2 x2 = {0.f, 0.f}, y2 = {0.f, 0.f}, z2 = {0.f, 0.f};
        double dx2 = 0.0, dy2 = 0.0, dz2 = 0.0;
        if constexpr (F64) {
            dx2 = P.r2[3 * (int64_t)jc];
            dy2 = P.r2[3 * (int64_t)jc + 1];
            dz2 = P.r2[3 * (int64_t)jc + 2];
        } else {
            x2 = P.r2d[jc];
            y2 = P.r2d[P.n2 + jc];
            z2 = P.r2d[2 * (int64_t)P.n2 + jc];
        }
        const float sa = F64 ? 0.f : pow2f(ea);
        auto mark = [&](int i, bool unsure) {
            const unsigned marks = __ballot_sync(0xffffffffu, unsure);
            if (lane == 0 && i < P.n1b && j < P.n2) {
                Q.marks[(int64_t)i * Q.mark_words + j / 32] = marks;
                if (marks)
                    *Q.marked = 1;
            }
        };
        const df::D a = df::make(P.a_ee_hi, P.a_ee_lo);
        for (int q = buf; q < ntiles; q += NB) {
            if (!tc::mbar_wait(tc::smem_u32(&tfull[buf]), (q / NB) & 1, s_abort)) {
                fail(16);
                break;
            }
            tc::fence_after_sync();
            const uint32_t cb = tbase + lane_off + (uint32_t)(Cfg::kBufCols * buf + R * pt0);
            const int i0 = (t_begin + q) * Cfg::kPts + pt0;  // r1 row of the tile
            if constexpr (F64) {
                double V[R];
                float lo[R], w[R];
                const float *bs = Q.bscale + (int64_t)i0 * R;
                const int *eb = Q.eb + (int64_t)i0 * R;
                const bool out = jok && i0 < P.n1b;
#pragma unroll
                for (int c = 0; c < R; c += 8) {
                    long long I[8];
                    float rest[8];
                    read_f64_8<S, BN>(cb + (uint32_t)c, I, rest);
                    float v[8];
                    tc::tmem_ld8(cb + (uint32_t)(BN * S + c), v);
                    if constexpr (PART) {
                        if (out)
#pragma unroll
                            for (int k = 0; k < 8; k++) {
                                const int64_t o = ((int64_t)i0 * R + c + k) * P.n2 + j;
                                if (!Q.first) {
                                    I[k] += Q.partI[o];
                                    rest[k] += Q.partL[o];
                                    v[k] += Q.partA[o];
                                }
                                if (!Q.last) {
                                    Q.partI[o] = I[k];
                                    Q.partL[o] = rest[k];
                                    Q.partA[o] = v[k];
                                }
                            }
                    }
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        scale_f64(I[k], rest[k], eb[c + k], ea, V + c + k, lo + c + k);
                        w[c + k] = bs[c + k] * fmaf(Q.check, v[k], -1.0f);
                    }
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0)
                    tc::mbar_arrive(tc::smem_u32(&tempty[buf]));
                if (!PART || Q.last)
                    mark(i0, out && (pair_f64<R>(Q, i0, j, V, lo, w, dx2, dy2, dz2) ||
                                     ea >= kNanExponent));
            } else {
                uint64_t H[R / 16][8], L[R / 16][8], L2[R / 16][8];
                float w[R];
#pragma unroll
                for (int h = 0; h < R / 16; h++) {
                    read_df16<S>(cb + 16u * h, H[h], L[h], L2[h]);
                    if constexpr (CHK) {
                        float v[16];
                        tc::tmem_ld16(cb + (uint32_t)(BN * S) + 16u * h, v);
#pragma unroll
                        for (int k = 0; k < 16; k++)
                            w[16 * h + k] = v[k];
                    }
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0)
                    tc::mbar_arrive(tc::smem_u32(&tempty[buf]));
                const bool out = jok && i0 < P.n1b;
                bool unsure = false;
                if (out) {
                    const float *bs = Q.bscale + (int64_t)i0 * R;
                    df::D V[R];
#pragma unroll
                    for (int h = 0; h < R / 16; h++)
                        scale_df16(H[h], L[h], L2[h], bs + 16 * h, V + 16 * h);
                    if constexpr (PART) {
#pragma unroll
                        for (int c = 0; c < R; c++) {
                            const int64_t at = ((int64_t)i0 * R + c) * P.n2 + j;
                            float2 *o = Q.part + at;
                            if (!Q.first)
                                V[c] = df::add(V[c], df::make(o->x, o->y));
                            if (!Q.last)
                                *o = make_float2(V[c].hi, V[c].lo);
                            if constexpr (CHK) {
                                if (!Q.first)
                                    w[c] += Q.partA[at];
                                if (!Q.last)
                                    Q.partA[at] = w[c];
                            }
                        }
                    }
                    if (!PART || Q.last) {
                        if constexpr (CHK)
#pragma unroll
                            for (int c = 0; c < R; c++)
                                w[c] = bs[c] * fmaf(Q.check, w[c], -1.0f);
                        unsure = pair_df<R, CHK>(Q, i0, j, V, w, x2, y2, z2, sa, a) ||
                                 (CHK && ea >= kNanExponent);
                    }
                }
                if constexpr (CHK)
                    if (!PART || Q.last)
                        mark(i0, unsure);
            }
        }
    }

    __syncwarp();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == kCtlWarp)
        tc::tmem_dealloc(tbase, kTmemCols);
}

// ---------------------------------------------------------------------------
// slicing of the operands
// ---------------------------------------------------------------------------

// Exponent e with |x| < 2^e for every x of the row; 0 for zero (or denormal-only) rows,
// kNanExponent for a row with an infinity or a NaN.
__device__ __forceinline__ int row_exponent(unsigned long long bits)
{
    const int E = (int)(bits >> 52);
    return E == 0 ? 0 : min(E - 1022, kNanExponent);
}

// slices[(s * Mpad + r) * Kpad + k] for r < Mpad, k < Kpad (a multiple of 32; zeros outside
// M x K), ex[r] = row exponent, of X[r * K + k]: one warp per row.  The digits are formed in
// integer arithmetic (digits.cuh).  kMag: the magnitudes on the row scale, truncated to BF16, as
// plane S.  scale (may be null): 2^ex[r], 0 for a zero row, with kMag NaN for rows beyond 2^100
// (which the check then leaves out).
template <int S, bool kMag>
__global__ void __launch_bounds__(256)
slice_kernel(const double *__restrict__ X, int M, int K, int Kpad, int Mpad,
             __nv_bfloat16 *__restrict__ slices, int *__restrict__ ex, float *__restrict__ scale)
{
    const int lane = threadIdx.x & 31;
    const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (r >= Mpad)
        return;
    unsigned long long m = 0;
    for (int k = lane; k < K && r < M; k += 32) {
        const unsigned long long v =
            (unsigned long long)__double_as_longlong(X[r * K + k]) & 0x7fffffffffffffffull;
        m = v > m ? v : m;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, o);
        m = v > m ? v : m;
    }
    const int e = row_exponent(m);
    if (lane == 0) {
        ex[r] = e;
        if (scale)
            scale[r] = (m >> 52) == 0 ? 0.0f : pow2f(kMag && e > 100 ? kNanExponent : e);
    }
    for (int k = lane; k < Kpad; k += 32) {
        const double x = r < M && k < K && e < kNanExponent ? X[r * K + k] : 0.0;
        int q[S];
        digits::digits_int<S>(digits::scaled_round<S>(x, e), q);
#pragma unroll
        for (int s = 0; s < S; s++)
            slices[((int64_t)s * Mpad + r) * Kpad + k] =
                __float2bfloat16_rn(__int2float_rn(q[s]) * exp2f((float)(-8 - 9 * s)));
        if constexpr (kMag) {
            const unsigned long long b = (unsigned long long)__double_as_longlong(x);
            const int E = (int)(b >> 52 & 0x7ff) - 1023 - e + 127;
            slices[((int64_t)S * Mpad + r) * Kpad + k] = __ushort_as_bfloat16(
                (unsigned short)(E > 0 ? (unsigned)E << 7 | ((unsigned)(b >> 45) & 0x7fu) : 0u));
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

static inline int64_t round_up(int64_t a, int64_t b) { return (a + b - 1) / b * b; }

// K of unchecked double-float contractions: 20 nuclei of 4 powers.
constexpr int kPlainDfK = 80;
// The K of one group in double-float: exact leading diagonals.
constexpr int kDfGroupK = 85;

// The K up to which the contraction is one group: the leading diagonals are exact (and the
// operands fit shared memory).  A longer one runs in groups of kGroupBlocks K blocks whose
// values are added between launches.
constexpr int kGroupBlocks = 2;
static int one_group_k(const PairTcMode &m) { return m.fp64 ? 64 : m.checked ? kDfGroupK : kPlainDfK; }
static int64_t pad_k(const PairTcMode &m, int64_t K)
{
    return round_up(std::max<int64_t>(K, 1), K <= one_group_k(m) ? kBK : kGroupBlocks * kBK);
}

static int planes(const PairTcMode &m) { return m.slices + (m.checked ? 1 : 0); }
// of a value between the groups: FP64 or double-float, and the magnitudes' sum
static int part_bytes(const PairTcMode &m) { return m.fp64 ? 16 : 12; }
static int mark_words(int64_t n2) { return (int)((n2 + 31) / 32); }


PairTcMode pair_tc_mode(const double *coef, const int *exps, int n_terms, int n_nuc, bool fp64,
                        int slices)
{
    PairTcMode m;
    m.fp64 = fp64;
    if (!fp64 && (getenv("CUTC_PAIR_DF") || getenv("CUTC_PAIR_DENSE")))
        return m;
    for (int k = 0; k < 3 * n_terms; k++)
        if (!std::isfinite(coef[k]))
            return m;
    m.rows = pair_df_sparse(exps, n_terms) ? 16 : 32;
    const int K = m.powers() * n_nuc;
    m.checked = fp64 || m.rows == 32 || K > kPlainDfK;
    // 32 rows of double-float values a pair between groups of K cost more than the loop over the
    // nuclei (2003 x 30 011 pairs: 57 ms in two groups, 110 in three; the loop 38, 46 and 96 ms
    // with 13, 16 and 24 nuclei)
    if (!fp64 && m.rows == 32 && K > kDfGroupK)
        return PairTcMode{};
    // Few nuclei with general exponents: where every term vanishes at its nucleus a large part
    // of the pairs is marked, and forming them again costs more than the loops over all pairs
    // (2003 x 30 011 pairs, 11 terms, double-float: one nucleus 9.8 to 14.3 ms, the loop 3.8; two
    // 4.0 with powers 0 among the terms, 7.1 to 10.5 without, the loop 6.3; three at most 6.0, the
    // loop 8.9.  512 x 20 011 in FP64: one nucleus 2.6 with powers 0, 3.4 to 3.7 without, the
    // loop 3.0; two at most 3.1, the loop 4.9)
    bool vanish = true;
    for (int k = 0; k < n_terms; k++)
        vanish = vanish && (exps[k] & 7) && (exps[k] >> 3 & 7);
    if (m.rows == 32 && ((n_nuc == 1 && (!fp64 || vanish)) || (n_nuc == 2 && !fp64 && vanish)))
        return PairTcMode{};
    // 5 slices (representation error 2^-45, under the error of a 5-slice build's operands), 6
    // for builds of 6 and 7 slices and where the check is (2^-54, below the double-float
    // epilogue), 7 for FP64 (2^-63)
    m.slices = fp64 ? 7 : slices >= 6 || m.checked ? 6 : 5;
    return m;
}

// Device bytes: per r2 point and r1 row, of K values in FP64 and in slices (and magnitudes).
static size_t operand_bytes(int64_t rows, int64_t K, int slices)
{
    return (size_t)rows * (8 * K + 2 * (slices + 1) * round_up(K, kGroupBlocks * kBK) + 4);
}

// r1 rows per sub-tile: its coefficient operand, and in groups its values so far, take about
// `limit` bytes each at most (eight rows at least).
static int64_t sub_tile_rows(const PairTcMode &m, int64_t n2, int64_t K, int64_t n1b, size_t limit)
{
    size_t per = operand_bytes(m.rows, K, m.slices);
    if (K > one_group_k(m))
        per = std::max<size_t>(per, (size_t)n2 * m.rows * part_bytes(m));
    return std::min(n1b, std::max<int64_t>(8, (int64_t)(limit / per) / 8 * 8));
}

static size_t sub_tile_bytes(size_t scratch) { return std::min(kPairScratch, scratch); }

size_t pair_tc_fixed_bytes(int n2, int n_nuc, int slices, size_t scratch)
{
    const int64_t K = 7 * (int64_t)n_nuc;
    size_t b = operand_bytes(round_up(n2, kBM), K, slices);
    if (K > 64)  // the values so far of a sub-tile
        b += std::max(sub_tile_bytes(scratch), (size_t)n2 * 8 * 32 * 16);
    return b;
}

int pair_tc_window(const PairTcMode &m, int n_nuc)
{
    const size_t per = operand_bytes(kBM, (int64_t)m.powers() * n_nuc, m.slices);
    return kBM * (int)std::max<size_t>(1, kPairScratch / per);
}

size_t pair_tc_row_bytes(int n_nuc, int slices)
{
    return operand_bytes(32, std::min<int64_t>(7 * (int64_t)n_nuc, 85), slices) + 3 * 8 + 32 * 4 + 64;
}

static int alloc_operand(Workspace &W, int slot, int S, int64_t M, int row_mult, int64_t K,
                         int64_t Kpad, SliceOperand &op)
{
    op.M = (int)M;
    op.Mpad = (int)round_up(std::max<int64_t>(M, 1), row_mult);
    op.K = K;
    op.Kpad = Kpad;
    void *p;
    CUTC_TRY(W.get(slot, (size_t)S * op.Mpad * op.Kpad * 2, &p));
    op.sl = p;
    CUTC_TRY(W.get(slot + 1, (size_t)op.Mpad * 4, &p));
    op.ex = (int *)p;
    return CUTC_OK;
}

template <int S, bool kMag>
static int slice_rows(cudaStream_t st, const double *X, const SliceOperand &op, float *scale)
{
    slice_kernel<S, kMag><<<ceil_div(op.Mpad, 8), 256, 0, st>>>(
        X, op.M, (int)op.K, (int)op.Kpad, op.Mpad, (__nv_bfloat16 *)op.sl, op.ex, scale);
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    return CUTC_OK;
}

static int slice_rows(cudaStream_t st, const PairTcMode &m, const double *X,
                      const SliceOperand &op, float *scale)
{
    return m.slices == 7 ? slice_rows<7, true>(st, X, op, scale)
           : m.checked   ? slice_rows<6, true>(st, X, op, scale)
           : m.slices == 6 ? slice_rows<6, false>(st, X, op, scale)
                           : slice_rows<5, false>(st, X, op, scale);
}

enum { kSlotAF = 0, kSlotBC = 2, kSlotF64 = 4, kSlotC64, kSlotR1d, kSlotBscale, kSlotPart, kSlotMarks };

int pair_tc_prepare(Workspace &W, int slot0, cudaStream_t st, const PairTcMode &mode, int n2,
                    int n_nuc, const double *f2, int64_t n1t, size_t scratch, int *err,
                    PairTcPlan &plan)
{
    const int64_t K = (int64_t)mode.powers() * n_nuc, Kpad = pad_k(mode, K);
    plan.mode = mode;
    plan.err = err;
    plan.tile_rows = sub_tile_rows(mode, n2, K, n1t, sub_tile_bytes(scratch));
    const int64_t rows = (int64_t)mode.rows * plan.tile_rows;
    void *p;
    CUTC_TRY(W.get(slot0 + kSlotF64, (size_t)n2 * K * 8, &p));
    plan.Fd = (double *)p;
    CUTC_TRY(W.get(slot0 + kSlotC64, (size_t)rows * K * 8, &p));
    plan.Cd = (double *)p;
    CUTC_TRY(W.get(slot0 + kSlotR1d, (size_t)3 * plan.tile_rows * sizeof(float2), &p));
    plan.r1d = (float2 *)p;
    CUTC_TRY(W.get(slot0 + kSlotBscale, (size_t)round_up(rows, kPairBN) * 4, &p));
    plan.bscale = (float *)p;
    if (K > one_group_k(mode)) {
        CUTC_TRY(W.get(slot0 + kSlotPart, (size_t)n2 * rows * part_bytes(mode), &p));
        plan.part = p;
    }
    if (mode.checked) {
        CUTC_TRY(W.get(slot0 + kSlotMarks, 64 + (size_t)plan.tile_rows * mark_words(n2) * 4, &p));
        plan.marked = (int *)p;
    }
    CUTC_TRY(alloc_operand(W, slot0 + kSlotAF, planes(mode), n2, kBM, K, Kpad, plan.AF));
    CUTC_TRY(alloc_operand(W, slot0 + kSlotBC, planes(mode), rows, kPairBN, K, Kpad, plan.BC));
    CUTC_TRY(launch_pair_tc_f(st, mode.powers(), n2, n_nuc, f2, plan.Fd));
    note_launches(1);
    return slice_rows(st, mode, plan.Fd, plan.AF, nullptr);
}

// 2-D map over slices [rows_total][Kpad] BF16, box = kBK x box_rows, 64B swizzle.
static int make_tmap(CUtensorMap *map, const void *base, int64_t rows_total, int64_t Kpad,
                     int box_rows)
{
    const uint64_t dims[2] = {(uint64_t)Kpad, (uint64_t)rows_total};
    const uint64_t strides[1] = {(uint64_t)Kpad * 2};
    const uint32_t box[2] = {(uint32_t)kBK, (uint32_t)box_rows};
    return encode_bf16_map(map, base, 2, dims, strides, box, 64);
}

template <int S, int KB, int R, bool F64, bool CHK, bool PART>
static int launch_kernel(cudaStream_t st, const CUtensorMap &ta, const CUtensorMap &tb,
                         PairTcParams Q, int n_sm)
{
    using Cfg = PairTcCfg<S, KB, R, F64, CHK>;
    static std::atomic<unsigned long long> attr_done{0};
    const unsigned long long bit = current_device_bit();
    if (!(attr_done.load() & bit)) {
        CUTC_CUDA_TRY(cudaFuncSetAttribute(pair_tc_kernel<S, KB, R, F64, CHK, PART>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem));
        attr_done.fetch_or(bit);
    }
    // CTAs that each walk a run of N tiles with their F tile resident: about eight per SM,
    // down to one per SM where that leaves a CTA fewer than 16 tiles to hide its set-up
    // behind (210 x 805 pairs in FP64: 47 us in 735 CTAs of 2 tiles)
    const int64_t all = (int64_t)Q.tiles_m * Q.tiles_n;
    const int64_t want = std::min<int64_t>(8, std::max<int64_t>(1, all / (16 * (int64_t)n_sm))) * n_sm;
    const int64_t chunks = std::max<int64_t>(
        1, std::min<int64_t>(Q.tiles_n, (want + Q.tiles_m - 1) / Q.tiles_m));
    Q.chunk = (int)((Q.tiles_n + chunks - 1) / chunks);
    const int64_t grid = (int64_t)Q.tiles_m * ((Q.tiles_n + Q.chunk - 1) / Q.chunk);
    if (grid > INT32_MAX) {
        cutc_set_error(CUTC_ERR_INVALID, "pair grid of %lld CTAs", (long long)grid);
        return CUTC_ERR_INVALID;
    }
    pair_tc_kernel<S, KB, R, F64, CHK, PART><<<(unsigned)grid, Cfg::kThreads, Cfg::kSmem, st>>>(ta, tb, Q);
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    return CUTC_OK;
}

template <int S, int R, bool F64, bool CHK>
static int launch_kb(cudaStream_t st, const CUtensorMap &ta, const CUtensorMap &tb,
                     const PairTcParams &Q, int n_sm, int KB, bool part)
{
    if constexpr (F64 || (CHK && R == 16))
        if (part)
            return launch_kernel<S, kGroupBlocks, R, F64, CHK, true>(st, ta, tb, Q, n_sm);
    if constexpr (F64 || !CHK || R == 32) {  // (others have more than 80 K)
        if (KB == 1)
            return launch_kernel<S, 1, R, F64, CHK, false>(st, ta, tb, Q, n_sm);
        if (KB == 2)
            return launch_kernel<S, 2, R, F64, CHK, false>(st, ta, tb, Q, n_sm);
    }
    if constexpr (!F64)
        if (KB == 3)
            return launch_kernel<S, 3, R, F64, CHK, false>(st, ta, tb, Q, n_sm);
    cutc_set_error(CUTC_ERR_INVALID, "pair contraction of %d K blocks", KB);
    return CUTC_ERR_INVALID;
}

// The tile's coefficient operand, then the kernel.
static int run_tile(cudaStream_t st, PairTcPlan &plan, PairTcParams Q, const double *rn,
                    double a_en, int n_sm)
{
    const PairTcMode &m = plan.mode;
    const PairDfArgs &P = Q.P;
    CUTC_TRY(launch_pair_tc_coef(st, m.rows, P.i0, P.n1b, P.nN, P.r1, rn, a_en, P.coef, P.exps,
                                 P.term_off, plan.Cd, plan.r1d));
    note_launches(1);
    SliceOperand B = plan.BC;
    B.M = m.rows * P.n1b;
    B.Mpad = (int)round_up(B.M, kPairBN);
    CUTC_TRY(slice_rows(st, m, plan.Cd, B, plan.bscale));
    CUtensorMap ta, tb;
    CUTC_TRY(make_tmap(&ta, plan.AF.sl, (int64_t)planes(m) * plan.AF.Mpad, plan.AF.Kpad, kBM));
    const int bn = m.fp64 ? m.rows : kPairBN;
    CUTC_TRY(make_tmap(&tb, B.sl, (int64_t)planes(m) * B.Mpad, B.Kpad, bn));
    Q.tiles_m = plan.AF.Mpad / kBM;
    Q.tiles_n = B.Mpad / bn;
    Q.chunk = 1;
    Q.Mpad = plan.AF.Mpad;
    Q.Npad = B.Mpad;
    Q.ea = plan.AF.ex;
    Q.eb = B.ex;
    Q.bscale = plan.bscale;
    Q.r1d = plan.r1d;
    Q.err = plan.err;
    const int KB = (int)(plan.AF.Kpad / kBK);
    const bool part = plan.AF.K > one_group_k(m);
    Q.part = (float2 *)plan.part;
    Q.partI = (long long *)plan.part;
    // the integers or double-float values, then (FP64) their rests, then the magnitudes' sums
    const int64_t part_n = part ? (int64_t)P.n2 * m.rows * P.n1b : 0;
    Q.partL = (float *)(Q.partI + part_n);
    Q.partA = Q.partL + (m.fp64 ? part_n : 0);
    Q.check = (m.fp64 ? 256.0f : 128.0f) / std::sqrt((float)plan.AF.K);
    Q.marked = plan.marked;
    Q.marks = (unsigned *)(plan.marked + 16);
    Q.mark_words = mark_words(P.n2);
    if (m.checked)
        CUTC_CUDA_TRY(cudaMemsetAsync(plan.marked, 0, sizeof(int), st));
    for (int kb = 0; kb < KB; kb += part ? kGroupBlocks : KB) {
        Q.kb0 = kb;
        Q.first = kb == 0;
        Q.last = !part || kb + kGroupBlocks >= KB;
        if (m.fp64 && m.rows == 16)
            CUTC_TRY((launch_kb<7, 16, true, true>(st, ta, tb, Q, n_sm, KB, part)));
        else if (m.fp64)
            CUTC_TRY((launch_kb<7, 32, true, true>(st, ta, tb, Q, n_sm, KB, part)));
        else if (m.rows == 32)
            CUTC_TRY((launch_kb<6, 32, false, true>(st, ta, tb, Q, n_sm, KB, part)));
        else if (m.checked)
            CUTC_TRY((launch_kb<6, 16, false, true>(st, ta, tb, Q, n_sm, KB, part)));
        else if (m.slices == 6)
            CUTC_TRY((launch_kb<6, 16, false, false>(st, ta, tb, Q, n_sm, KB, part)));
        else
            CUTC_TRY((launch_kb<5, 16, false, false>(st, ta, tb, Q, n_sm, KB, part)));
    }
    return CUTC_OK;
}

int pair_tc_tile_df(cudaStream_t st, PairTcPlan &plan, const PairDfArgs &P, const double *rn,
                    double a_en, int n_sm)
{
    if (P.n1b <= 0 || P.n2 <= 0)
        return CUTC_OK;
    for (int64_t i = 0; i < P.n1b; i += plan.tile_rows) {
        PairTcParams Q{};
        Q.P = P;
        Q.P.i0 += (int)i;
        Q.P.n1b = (int)std::min<int64_t>(plan.tile_rows, P.n1b - i);
        Q.P.G += i * P.ldg;
        CUTC_TRY(run_tile(st, plan, Q, rn, a_en, n_sm));
        if (plan.mode.checked) {
            PairArgs R{};
            R.i0 = Q.P.i0; R.n1b = Q.P.n1b; R.n2 = P.n2; R.nN = P.nN;
            R.r1 = P.r1; R.r2 = P.r2; R.f2 = P.f2;
            R.coef = P.coef; R.exps = P.exps; R.term_off = P.term_off; R.a_ee = P.a_ee;
            R.G = reinterpret_cast<double *>(Q.P.G); R.ldg = P.ldg; R.plane = P.plane;
            CUTC_TRY(launch_pair_f64_marked(st, R, rn, a_en, true, plan.marked,
                                            (const unsigned *)(plan.marked + 16), mark_words(P.n2),
                                            n_sm));
        }
    }
    return CUTC_OK;
}

int pair_tc_tile_f64(cudaStream_t st, PairTcPlan &plan, const PairArgs &A, const double *rn,
                     double a_en, int n_sm)
{
    if (A.n1b <= 0 || A.n2 <= 0)
        return CUTC_OK;
    PairTcParams Q{};
    PairDfArgs &P = Q.P;
    P.i0 = A.i0; P.n1b = A.n1b; P.n2 = A.n2; P.nN = A.nN;
    P.r1 = A.r1; P.r2 = A.r2; P.coef = A.coef; P.exps = A.exps; P.term_off = A.term_off;
    P.a_ee = A.a_ee; P.ldg = A.ldg; P.plane = A.plane;
    for (int64_t i = 0; i < A.n1b; i += plan.tile_rows) {
        P.i0 = A.i0 + (int)i;
        P.n1b = (int)std::min<int64_t>(plan.tile_rows, A.n1b - i);
        Q.G64 = A.G + i * A.ldg;
        CUTC_TRY(run_tile(st, plan, Q, rn, a_en, n_sm));
        PairArgs R = A;
        R.i0 = P.i0;
        R.n1b = P.n1b;
        R.G = Q.G64;
        CUTC_TRY(launch_pair_f64_marked(st, R, rn, a_en, false, plan.marked,
                                        (const unsigned *)(plan.marked + 16), mark_words(A.n2), n_sm));
    }
    return CUTC_OK;
}

}  // namespace cutc
