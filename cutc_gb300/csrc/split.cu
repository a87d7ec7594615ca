// The split form's contractions (modular.cu), its pair terms on the tensor cores
// (tcgen05 + TMA), and the operands of both.
//
// Both dense contractions of the cutc_int path
//   X_m[p, r1] = sum_r2 P[p, r2] G_m[r1, r2]                    (X build)
//   H[p, q] = sum_r1 X_3[p, r1] S0[q, r1],
//   N[p, l] = -1/2 sum_{m, r1} X_m[p, r1] S_m[l, r1]          (int_2e)
// are C[M x N] = alpha * A[M x K] B[N x K]^T with FP64 operands and run as modular
// contractions: exact integer products of the operands rounded on their row scales,
// one BF16 tensor-core product per modulus (moduli.cuh).  n_slices chooses the number of
// moduli (split_moduli): the precision of at least that many 9-bit slices.
//
// The pair terms' short contraction (K = 4 n_nuc) keeps the splitting into S slices,
//     A[r, k] = 2^{e_r} sum_{s < S} a_s[r, k],  a_s = q_s 2^{-8-9s},  q_s in [-256, 256]
// (S signed 9-bit digits of the row-scaled value), whose products a_s b_t, s + t < S,
// run as BF16 tcgen05.mma with one FP32 accumulator per diagonal s + t: with K <= 80 the
// leading diagonals are exact in FP32, and the S slices of b are read by one instruction
// per slice of a (the error-free splitting of Ozaki, Ogita, Oishi and Rump 2012).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <atomic>
#include <cstdlib>
#include <vector>

#include "common.cuh"
#include "dfloat.cuh"
#include "digits.cuh"
#include "pair.cuh"
#include "products.cuh"
#include "residue.cuh"
#include "split.cuh"
#include "tc.cuh"

namespace cutc {

constexpr int kBM = 128;        // rows of A per CTA (TMEM lanes)
constexpr int kBK = 32;         // K per TMA box: 32 BF16 = 64-byte rows (64B swizzle)
constexpr int kMaxKPerLaunch = 1 << 18;
// Default K per launch (one panel of residues): one launch up to kLongK; a longer
// contraction runs as equal launches of at most kLaunchK, whose residues are added up.
// With an A operand of kBigM rows or more, launches of at most kLaunchKBigM, which bound
// the residues of its panel.
constexpr int kLongK = 65536;
constexpr int kLaunchK = 49152;
constexpr int kBigM = 16384;
constexpr int kLongKBigM = 32768;
constexpr int kLaunchKBigM = 24576;
constexpr uint32_t kTmemCols = 512;

// ---------------------------------------------------------------------------
// Pair terms on the tensor cores (split form, Jastrow exponents in {0, 2, 3, 4})
//
// The nucleus sum of grad1 u(r1, r2) is, for fixed g12, the contraction
//   V_c(r1, r2) = sum_k C[(r1, c)][k] F[r2][k],  k = 4 A + q over (nucleus, power of f2)
// (pair_df.cu builds F and the 16 coefficient rows C per r1 point in FP64).  Here it
// runs as a split contraction: A = the F slices (one 128-row tile of r2 points, all
// of K, loaded once per CTA), B = the coefficient slices (N tiles of 64 rows = four
// r1 points, streamed), one stacked-diagonal accumulator set in tensor memory.  The
// tensor-core work of a tile is about 1/40 of its epilogue, so one accumulator set and
// one B stage suffice: the next tile's MMAs run as soon as the epilogue has read the
// accumulators, long before it needs them, and one control warp issues both the TMA
// loads and the MMAs, which leaves registers for 16 epilogue warps (4 per SM
// sub-partition) to hide the latency of their dependent double-float chains.
// K = 4 n_nuc <= 80, so every diagonal sum is one chunk:
// diagonals 0..2 are exact in FP32 ((d + 1) * 80 * 2^16 < 2^24), d >= 3 are 2^-27 and
// below, where FP32 rounding is immaterial.
//
// The epilogue warps (lane = r2 point, one r1 point per warp) read the S diagonals
// of the point's 16 columns, add them exactly on fixed grids into double-float
// values, release the accumulators, then finish the pair in double-float exactly as
// pair_df_kernel does: g12 and its gradient, the powers of
// g, -1/2 |grad u|^2, the FP64 path near e-e coalescence and the (hi, lo) G planes.  Per pair that is about 800 FP32 operations
// instead of 30 df multiply-adds (~450 operations) per nucleus.
// ---------------------------------------------------------------------------

struct PairTcParams {
    int tiles_m, tiles_n, chunk;  // r2 tiles of 128 points, N tiles, N tiles per CTA
    int Mpad, Npad;               // padded rows of the F and coefficient slices
    const int *ea;                // row exponents of the F slices
    const float *bscale;          // 2^(row exponent) of each coefficient row
    const float2 *r1d;            // the tile's r1 points in double-float, [3 i + c]
    PairDfArgs P;                 // geometry, near-coalescence path and outputs
    int *err;
};

// bscale[r] = 2^ex[r] as a float
__global__ void exp_scale_kernel(const int *__restrict__ ex, int rows, float *__restrict__ bscale)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < rows) {
        const int e = max(-126, min(127, ex[r]));
        bscale[r] = __int_as_float((e + 127) << 23);
    }
}

constexpr int kPairBN = 64;  // coefficient rows per N tile: four r1 points x 16 columns

template <int S, int KB>
struct PairTcCfg {
    static constexpr int kBN = kPairBN;
    static constexpr int kPts = kBN / 16;
    static constexpr int kEpiWarps = 4 * kPts;       // lane quarter x r1 point
    static constexpr int kCtlWarp = kEpiWarps;       // TMA loads and MMAs, lane 0
    static constexpr int kThreads = (kEpiWarps + 1) * 32;
    static constexpr int kASlice = kBM * kBK * 2;
    static constexpr int kBSlice = kBN * kBK * 2;
    static constexpr int kABytes = KB * S * kASlice;
    static constexpr int kBStage = KB * S * kBSlice;
    static constexpr int kSmem = kABytes + kBStage + 1024 + 256;
    static constexpr int kMaxN = 256;                // widest kind::f16 instruction at M = 128
    static_assert(kSmem <= 227 * 1024, "shared memory");
    static_assert(kBN * S <= (int)kTmemCols, "accumulators exceed tensor memory");
    static_assert(kMaxN % kBN == 0, "instruction splits on diagonal boundaries");
    static_assert(kBSlice % 512 == 0, "B slices must stack on 8-row swizzle atoms");
    // 17 warps: the compiler's register budget is 96 per thread (it rounds the warps of
    // a CTA up when it divides the register file)
    static_assert(kThreads <= 1024, "threads per CTA");
};

// x 2^e for the scale of a value of row exponents e (clamped to the float range)
__device__ __forceinline__ float pow2f(int e)
{
    e = e < -126 ? -126 : (e > 127 ? 127 : e);
    return __int_as_float((e + 127) << 23);
}

template <int S, int KB>
__global__ void __launch_bounds__(PairTcCfg<S, KB>::kThreads, 1)
pair_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ PairTcParams Q)
{
    using Cfg = PairTcCfg<S, KB>;
    constexpr int D = S - 1, BN = Cfg::kBN;
    constexpr int kEpiWarps = Cfg::kEpiWarps, kCtlWarp = Cfg::kCtlWarp;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem;
    uint8_t *sB = smem + Cfg::kABytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(sB + Cfg::kBStage);
    uint64_t *afull = bars;      // the F tile has landed
    uint64_t *full = bars + 1;   // the B stage holds tile q
    uint64_t *empty = bars + 2;  // the MMAs of tile q are done with the B stage
    uint64_t *tfull = bars + 3;  // the accumulators hold tile q
    uint64_t *tempty = bars + 4; // every epilogue warp has read tile q's accumulators
    uint64_t *drain = bars + 5;
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(drain + 1);
    volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);

    const PairDfArgs &P = Q.P;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = (int)(blockIdx.x % Q.tiles_m) * kBM;
    const int t_begin = (int)(blockIdx.x / Q.tiles_m) * Q.chunk;
    const int ntiles = min(Q.tiles_n, t_begin + Q.chunk) - t_begin;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 5; i++)
            tc::mbar_init(tc::smem_u32(&bars[i]), i == 4 ? kEpiWarps : 1);
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
            auto load_b = [&](int q) {
                const uint32_t fb = tc::smem_u32(full);
                tc::mbar_arrive_expect_tx(fb, Cfg::kBStage);
                const int n0 = (t_begin + q) * BN;
#pragma unroll
                for (int kb = 0; kb < KB; kb++)
#pragma unroll
                    for (int t = 0; t < S; t++)
                        tc::tma_load_2d(tc::smem_u32(sB + (kb * S + t) * Cfg::kBSlice), &tmB,
                                        kb * kBK, t * Q.Npad + n0, fb);
            };
            const uint32_t ab = tc::smem_u32(afull);
            tc::mbar_arrive_expect_tx(ab, Cfg::kABytes);
#pragma unroll
            for (int kb = 0; kb < KB; kb++)
#pragma unroll
                for (int s = 0; s < S; s++)
                    tc::tma_load_2d(tc::smem_u32(sA + (kb * S + s) * Cfg::kASlice), &tmA, kb * kBK,
                                    s * Q.Mpad + m0, ab);
            int loaded = 0;  // B tiles issued into the stage
            if (ntiles > 0) {
                load_b(0);
                loaded = 1;
            }
            bool ok = tc::mbar_wait(ab, 0, s_abort);
            if (!ok)
                fail(12);
            for (int q = 0; q < ntiles && ok; q++) {
                // the accumulators are free once every epilogue warp has read tile q - 1
                if (q >= 1 && !tc::mbar_wait(tc::smem_u32(tempty), (q - 1) & 1, s_abort)) {
                    fail(13);
                    break;
                }
                if (!tc::mbar_wait(tc::smem_u32(full), q & 1, s_abort)) {
                    fail(14);
                    break;
                }
                tc::fence_after_sync();
                const uint32_t sb0 = tc::smem_u32(sB);
                const uint32_t sa0 = tc::smem_u32(sA);
                bool first = true;
#pragma unroll
                for (int kb = 0; kb < KB; kb++) {
#pragma unroll
                    for (int k16 = 0; k16 < kBK / 16; k16++) {
#pragma unroll
                        for (int s = 0; s < S; s++) {
                            // a_s x [b_0 .. b_{D-s}] -> diagonals s .. D, in instructions of
                            // at most kMaxN columns
                            const uint64_t ad = tc::smem_desc_sw64(
                                sa0 + (kb * S + s) * Cfg::kASlice + k16 * 32);
#pragma unroll
                            for (int t0 = 0; t0 <= D - s; t0 += Cfg::kMaxN / BN) {
                                const int nt = min(Cfg::kMaxN / BN, D - s + 1 - t0);
                                const uint64_t bd = tc::smem_desc_sw64(
                                    sb0 + (kb * S + t0) * Cfg::kBSlice + k16 * 32);
                                tc::mma_bf16(tbase + (uint32_t)(BN * (s + t0)), ad, bd,
                                             tc::idesc_bf16_f32(kBM, BN * nt), first ? 0u : 1u);
                            }
                            first = false;
                        }
                    }
                }
                tc::mma_commit(tc::smem_u32(empty));
                tc::mma_commit(tc::smem_u32(tfull));
                // refill the B stage for tile q + 1 once these MMAs have read it
                if (q + 1 < ntiles) {
                    if (!tc::mbar_wait(tc::smem_u32(empty), q & 1, s_abort)) {
                        fail(11);
                        break;
                    }
                    load_b(q + 1);
                    loaded = q + 2;
                }
            }
            tc::mma_commit(tc::smem_u32(drain));
            if (!tc::mbar_wait(tc::smem_u32(drain), 0, nullptr))
                fail(15);
            // let the copies still in flight land before the CTA goes away
            tc::mbar_wait(ab, 0, nullptr);
            if (*s_abort && loaded > 0)
                tc::mbar_wait(tc::smem_u32(full), (loaded - 1) & 1, nullptr);
        }
    } else {
        // ---- epilogue: one r1 point of each N tile, 32 r2 points ---------------------
        const int quarter = warp & 3, pt = warp >> 2;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        const int j = m0 + quarter * 32 + lane;
        const bool jok = j < P.n2;
        const int jc = jok ? j : 0;
        const float2 x2 = P.r2d[jc], y2 = P.r2d[P.n2 + jc], z2 = P.r2d[2 * (int64_t)P.n2 + jc];
        const float sa = pow2f(Q.ea[jc]);  // F rows: 2^1 (f^0 = 1 is the row maximum)
        const df::D a = df::make(P.a_ee_hi, P.a_ee_lo);
        for (int q = 0; q < ntiles; q++) {
            if (!tc::mbar_wait(tc::smem_u32(tfull), q & 1, s_abort)) {
                fail(16);
                break;
            }
            tc::fence_after_sync();
            // The point's 16 columns on each diagonal, summed exactly on grids.  In units of
            // the row scales every diagonal sum D_d is a multiple of 2^(-16-9d) and |D_0| <= K:
            //   H  = D_0 + D_1 rounded to multiples of 2^-16      (exact: below 2^7 there)
            //   L  = the rest of D_1 + D_2 rounded to 2^-25         (exact: below 2^-8 there)
            //   L2 = the rest of D_2 + D_3 + ... (FP32; below 2^-18, so off by < 2^-42)
            // Two columns share each packed f32x2 operation.
            uint64_t H[8], L[8], L2[8];
            {
                const uint32_t cb = tbase + lane_off + (uint32_t)(16 * pt);
                const uint64_t C16 = tc::f2_pack(__float_as_uint(192.0f), __float_as_uint(192.0f));
                const uint64_t C25 = tc::f2_pack(__float_as_uint(0.375f), __float_as_uint(0.375f));
                float v[16];
                tc::tmem_ld16(cb, v);
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    H[k] = tc::f2_pack(__float_as_uint(v[2 * k]), __float_as_uint(v[2 * k + 1]));
                    L[k] = L2[k] = 0ull;
                }
#pragma unroll
                for (int d = 1; d <= D; d++) {
                    tc::tmem_ld16(cb + (uint32_t)(BN * d), v);
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const uint64_t x =
                            tc::f2_pack(__float_as_uint(v[2 * k]), __float_as_uint(v[2 * k + 1]));
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
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0)
                tc::mbar_arrive(tc::smem_u32(tempty));

            const int i = (t_begin + q) * Cfg::kPts + pt;  // r1 row of the tile
            if (i >= P.n1b)
                continue;
            // V_c 2^-ea = 2^eb_c ((H + L) + L2): TwoSum of H and L, then the rest.  The F
            // rows' scale 2^ea, a power of two common to the 16 values, multiplies the
            // results instead (the polynomial is linear in V, and power-of-two scaling
            // commutes with the double-float arithmetic).
            df::D V[16];
            const float *scr = Q.bscale + (int64_t)i * 16;  // 16-float aligned rows
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
            const int64_t o = (int64_t)i * P.ldg + j;
            if (jok) {
                float2 w4[4];
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
                const df::D g2 = df::sqr(g);
                // sum_o g^o V_o, o = 0, 2, 3, 4
                df::D ux = df::fma(df::fma(df::fma(V[3], g, V[2]), g, V[1]), g2, V[0]);
                df::D uy = df::fma(df::fma(df::fma(V[7], g, V[6]), g, V[5]), g2, V[4]);
                df::D uz = df::fma(df::fma(df::fma(V[11], g, V[10]), g, V[9]), g2, V[8]);
                const df::D dudg = df::mul(df::fma(df::fma(V[14], g, V[13]), g, V[12]), g);
                ux = df::fma(dudg, gx, ux);
                uy = df::fma(dudg, gy, uy);
                uz = df::fma(dudg, gz, uz);
                ux = df::make(__fmul_rn(ux.hi, sa), __fmul_rn(ux.lo, sa));
                uy = df::make(__fmul_rn(uy.hi, sa), __fmul_rn(uy.lo, sa));
                uz = df::make(__fmul_rn(uz.hi, sa), __fmul_rn(uz.lo, sa));
                const df::D n2v = df::add(df::add(df::sqr(ux), df::sqr(uy)), df::sqr(uz));
                const df::D lv = df::mul_f(n2v, -0.5f);
                w4[0] = make_float2(ux.hi, ux.lo);
                w4[1] = make_float2(uy.hi, uy.lo);
                w4[2] = make_float2(uz.hi, uz.lo);
                w4[3] = make_float2(lv.hi, lv.lo);
#pragma unroll
                for (int c = 0; c < 4; c++)
                    P.G[o + c * P.plane] = w4[c];
            }
        }
    }

    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == kCtlWarp)
        tc::tmem_dealloc(tbase, kTmemCols);
}

// ---------------------------------------------------------------------------
// slicing kernels
// ---------------------------------------------------------------------------

// wchi[a * n + g] = w[g] chi_a(g), chi_a at chi[a * ldchi]
__global__ void weighted_aos_kernel(int n, const double *__restrict__ w,
                                    const double *__restrict__ chi, int64_t ldchi,
                                    double *__restrict__ wchi)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int a = blockIdx.y;
    if (g < n)
        wchi[(int64_t)a * n + g] = w[g] * chi[(int64_t)a * ldchi + g];
}

static int weighted_aos(cudaStream_t st, int n, int nA, const double *w, const double *chi,
                        int64_t ldchi, double *wchi)
{
    if (n <= 0 || nA <= 0)
        return CUTC_OK;
    weighted_aos_kernel<<<dim3(ceil_div(n, 256), nA), 256, 0, st>>>(n, w, chi, ldchi, wchi);
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    return CUTC_OK;
}

// |v| as its bits; NaN counts as 0, as fmax would skip it.  Integer work: an FP64 max
// would take the FP64 pipe.
__device__ __forceinline__ unsigned long long max_bits(double v)
{
    const unsigned long long b = abs_bits(v);
    return b > 0x7ff0000000000000ull ? 0ull : b;
}

// rmax[r] = bits of max_k |src(r, k)|
template <class Src>
__global__ void rowmax_kernel(Src src, int rows, int64_t K, int64_t kper,
                              unsigned long long *rmax)
{
    const int r = blockIdx.x;
    if (r >= rows)
        return;
    const int64_t k0 = (int64_t)blockIdx.y * kper;
    const int64_t k1 = min(K, k0 + kper);
    unsigned long long m = 0;
    for (int64_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const unsigned long long b = max_bits(src(r, k));
        m = b > m ? b : m;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long b = __shfl_xor_sync(0xffffffffu, m, o);
        m = b > m ? b : m;
    }
    __shared__ unsigned long long red[32];
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long b = __shfl_xor_sync(0xffffffffu, m, o);
            m = b > m ? b : m;
        }
        if (threadIdx.x == 0 && m > 0)
            atomicMax(&rmax[r], m);
    }
}

// Exponent e with |x| < 2^e for every x of the row; 0 for zero (or denormal-only) rows.
__device__ __forceinline__ int row_exponent(unsigned long long bits)
{
    const int E = (int)((bits >> 52) & 0x7ff);
    return E == 0 ? 0 : E - 1022;
}

// The S signed base-2^9 digits of t (digits.cuh) as exact BF16 values q_s 2^{-8-9s}.
template <int S>
__device__ __forceinline__ void digits_of(long long t, __nv_bfloat16 (&out)[S])
{
    int q[S];
    digits::digits_int<S>(t, q);
#pragma unroll
    for (int s = 0; s < S; s++)
        out[s] = __float2bfloat16_rn(__int2float_rn(q[s]) * exp2f((float)(-8 - 9 * s)));
}

// The digits of an FP64 value x 2^{-e} (first digit scaled by 2^8).
template <int S>
__device__ __forceinline__ void split_digits(double x, int e, __nv_bfloat16 (&out)[S])
{
    digits_of<S>(digits::scaled_round<S>(x, e), out);
}

// slices[(s * Mpad + r) * Kpad + k] for r < Mpad, k < Kpad (zeros outside M x K);
// ex[r] = row exponent.  Four consecutive k per thread (Kpad is a multiple of 32),
// so each slice plane gets one 8-byte store per thread.  Rows are taken
// blockIdx.y, blockIdx.y + gridDim.y, ...: any row count fits the grid.
template <int S, class Src>
__global__ void slice_kernel(Src src, int M, int64_t K, int64_t Kpad, int Mpad,
                             const unsigned long long *rmax, __nv_bfloat16 *slices, int *ex)
{
    const int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (k >= Kpad)
        return;
    for (int r = blockIdx.y; r < Mpad; r += gridDim.y) {
        const int e = r < M ? row_exponent(rmax[r]) : 0;
        if (k == 0)
            ex[r] = e;
        __nv_bfloat16 d[4][S];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const double x = (r < M && k + q < K) ? src(r, k + q) : 0.0;
            split_digits<S>(x, e, d[q]);
        }
#pragma unroll
        for (int s = 0; s < S; s++) {
            __nv_bfloat162 lo, hi;
            lo.x = d[0][s];
            lo.y = d[1][s];
            hi.x = d[2][s];
            hi.y = d[3][s];
            uint2 w;
            w.x = *reinterpret_cast<unsigned *>(&lo);
            w.y = *reinterpret_cast<unsigned *>(&hi);
            *reinterpret_cast<uint2 *>(slices + ((int64_t)s * Mpad + r) * Kpad + k) = w;
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

static inline int64_t round_up(int64_t a, int64_t b) { return (a + b - 1) / b * b; }

// 2-D map over slices [rows_total][Kpad] BF16, box = kBK x box_rows, 64B swizzle.
static int make_tmap(CUtensorMap *map, const void *base, int64_t rows_total, int64_t Kpad,
                     int box_rows)
{
    const uint64_t dims[2] = {(uint64_t)Kpad, (uint64_t)rows_total};
    const uint64_t strides[1] = {(uint64_t)Kpad * 2};
    const uint32_t box[2] = {(uint32_t)kBK, (uint32_t)box_rows};
    return encode_bf16_map(map, base, 2, dims, strides, box, 64);
}

static int alloc_operand(Workspace &W, int slot, int S, int M, int row_mult, int64_t K,
                         Operand &op)
{
    op.M = M;
    op.Mpad = (int)round_up(std::max(M, 1), row_mult);
    op.K = K;
    op.Kpad = round_up(std::max<int64_t>(K, 1), kBK);
    void *p;
    CUTC_TRY(W.get(slot, (size_t)S * op.Mpad * op.Kpad * 2, &p));
    op.sl = p;
    CUTC_TRY(W.get(slot + 1, (size_t)op.Mpad * 4, &p));
    op.ex = (int *)p;
    CUTC_TRY(W.get(slot + 2, (size_t)op.Mpad * 8, &p));
    op.rmax = (unsigned long long *)p;
    return CUTC_OK;
}

template <int S, class Src>
static int slice_rows(cudaStream_t st, Src src, Operand &op)
{
    CUTC_CUDA_TRY(cudaMemsetAsync(op.rmax, 0, (size_t)op.Mpad * 8, st));
    if (op.M > 0 && op.K > 0) {
        const int64_t kper = 16384;
        dim3 g1((unsigned)op.M, ceil_div(op.K, kper));
        rowmax_kernel<Src><<<g1, 256, 0, st>>>(src, op.M, op.K, kper, op.rmax);
        CUTC_CUDA_TRY(cudaGetLastError());
    }
    if (op.Kpad % 4) {
        cutc_set_error(CUTC_ERR_INVALID, "operand K padding %lld is not a multiple of 4",
                       (long long)op.Kpad);
        return CUTC_ERR_INVALID;
    }
    dim3 g2(ceil_div(op.Kpad, 4 * 256), (unsigned)std::min(op.Mpad, 65535));
    slice_kernel<S, Src><<<g2, 256, 0, st>>>(src, op.M, op.K, op.Kpad, op.Mpad, op.rmax,
                                             (__nv_bfloat16 *)op.sl, op.ex);
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(2);
    return CUTC_OK;
}

int split_k_blocks_per_launch(int64_t K, int64_t M, int k_split)
{
    const int64_t nkb_total = (std::max<int64_t>(K, 1) + kBK - 1) / kBK;
    if (k_split > 0)
        return std::max(1, std::min(k_split, kMaxKPerLaunch) / kBK);
    const int64_t kt = nkb_total * kBK;
    const bool big = M >= kBigM;
    const int64_t one = big ? kLongKBigM : kLongK, each = big ? kLaunchKBigM : kLaunchK;
    const int64_t launches = kt <= one ? 1 : (kt + each - 1) / each;
    return (int)((nkb_total + launches - 1) / launches);
}

// ---------------------------------------------------------------------------
// the plan for one build
// ---------------------------------------------------------------------------

enum SplitSlot {
    SS_PAIRS_SYM = 0, SS_PAIRS_ANTI, SS_ERR,
    SS_AX, SS_AX_SC, SS_BX, SS_BX_SC, SS_RES,              // X build
    SS_AI, SS_AI_SC, SS_BH, SS_BH_SC, SS_BN, SS_BN_SC,     // int_2e
    SS_AF, SS_BC = SS_AF + 3, SS_F64 = SS_BC + 3, SS_C64, SS_R1D, SS_BSCALE,  // pair terms
    SS_WCHI2, SS_WCHI1,
};

// K panel of a contraction (one launch's K).
static int64_t panel_k(int64_t K, int64_t M, int k_split)
{
    return std::min(K, (int64_t)split_k_blocks_per_launch(K, M, k_split) * kBK);
}

// Device bytes for the residues of B's columns: as many as the G tile they are formed
// from takes (its rows are then read once per panel, in a few groups of columns), at
// least 1 GiB, so that small contractions run in one group.
constexpr size_t kMinResidueBytes = (size_t)1 << 30;
static size_t x_residue_bytes(int64_t rows, int64_t n2)
{
    return std::max(kMinResidueBytes, (size_t)rows * 4 * (size_t)n2 * 8);
}
// Device bytes of each operand's residues in the int_2e contractions.
constexpr size_t kInt2eResidueBytes = (size_t)4 << 30;

// K panel of the int_2e contractions: whole tensor-core chunks (256) whose residues of the
// np rows of A fit.
static int64_t int2e_panel_k(int n_mod, int64_t K, int64_t np, int k_split)
{
    const int64_t fit = (int64_t)(kInt2eResidueBytes / (2 * (size_t)n_mod * np)) / 256 * 256;
    const int64_t cap = k_split > 0 ? panel_k(K, np, k_split) : K;
    return std::min(cap, std::max<int64_t>(256, fit));
}

size_t split_r1_row_bytes(const Request &R)
{
    return 4 * (size_t)R.n2 * 8 + 64;  // residues, as many bytes as the four G rows
}

size_t split_int2e_row_bytes(const Request &R)
{
    return 8 * (size_t)R.nA + 64;  // the point's weighted AO values w chi_a
}

size_t split_fixed_bytes(const Request &R)
{
    // residues of a K panel of P, the weighted AO values w chi_a on r2 they are formed
    // from, the int_2e operands' residues, and the residues of one pass of results
    const int n_mod = split_moduli(R.n_slices);
    const int64_t np = n_pairs(R.nA);
    size_t b = residue_bytes(n_mod, np, panel_k(R.n2, np, R.k_split)) + 8 * (size_t)R.nA * R.n2 +
               std::min(kMinResidueBytes, residue_bytes(n_mod, 4 * (int64_t)R.n1, R.n2)) +
               modular_out_bytes(n_mod, np,
                                 std::max<int64_t>(np, std::min<int64_t>(4 * (int64_t)R.n1, 1 << 30)));
    if (!R.x_only)
        b += std::min(kInt2eResidueBytes, residue_bytes(n_mod, np, 3 * (int64_t)R.n1)) * 3;
    return b;
}

static int upload_pairs(Workspace &W, int slot, cudaStream_t st, int nA, bool strict, int2 **out)
{
    std::vector<int2> v;
    for (int b = 0; b < nA; b++)
        for (int a = strict ? b + 1 : b; a < nA; a++)
            v.push_back(make_int2(a, b));  // packed order of tri_index / stri_index
    void *p;
    CUTC_TRY(W.get(slot, std::max<size_t>(1, v.size()) * sizeof(int2), &p));
    if (!v.empty())
        CUTC_CUDA_TRY(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(int2), cudaMemcpyHostToDevice, st));
    CUTC_CUDA_TRY(cudaStreamSynchronize(st));  // v goes out of scope
    *out = (int2 *)p;
    return CUTC_OK;
}

#define CUTC_SLICES_DISPATCH(S_, CALL)                                         \
    switch (S_) {                                                              \
    case 3: { constexpr int S = 3; CALL; } break;                              \
    case 4: { constexpr int S = 4; CALL; } break;                              \
    case 5: { constexpr int S = 5; CALL; } break;                              \
    case 6: { constexpr int S = 6; CALL; } break;                              \
    case 7: { constexpr int S = 7; CALL; } break;                              \
    default:                                                                   \
        cutc_set_error(CUTC_ERR_INVALID, "unsupported slice count %d", S_);    \
        return CUTC_ERR_INVALID;                                               \
    }

// Row scales of an operand.
static int scale_slot(Workspace &W, int slot, int rows, int **sc)
{
    void *p;
    CUTC_TRY(W.get(slot, std::max<size_t>(1, rows) * sizeof(int), &p));
    *sc = (int *)p;
    return CUTC_OK;
}

int split_prepare_x(Engine *E, const Request &R, cudaStream_t st, const double *wr2,
                    const double *aos2v, int64_t n1t, int slot0, SplitPlan &sp)
{
    Workspace &W = E->ws;
    sp.slot0 = slot0;
    sp.n_slices = R.n_slices;
    sp.n1t = n1t;
    const int n_mod = split_moduli(R.n_slices);
    const int np = (int)n_pairs(R.nA);
    void *p;
    CUTC_TRY(W.get(slot0 + SS_ERR, 64, &p));
    sp.err = (int *)p;
    CUTC_CUDA_TRY(cudaMemsetAsync(sp.err, 0, 4, st));
    CUTC_TRY(upload_pairs(W, slot0 + SS_PAIRS_SYM, st, R.nA, false, &sp.pairs_sym));
    CUTC_TRY(upload_pairs(W, slot0 + SS_PAIRS_ANTI, st, R.nA, true, &sp.pairs_anti));
    CUTC_TRY(scale_slot(W, slot0 + SS_AX_SC, np, &sp.sc_ax));
    CUTC_TRY(scale_slot(W, slot0 + SS_BX_SC, (int)(4 * n1t), &sp.sc_bx));
    sp.k_panel = panel_k(R.n2, np, R.k_split);
    CUTC_TRY(W.get(slot0 + SS_AX, residue_bytes(n_mod, np, sp.k_panel), &p));
    sp.ax.p = p;
    sp.ax.rows = np;
    CUTC_TRY(W.get(slot0 + SS_WCHI2, std::max<size_t>(1, (size_t)R.nA * R.n2) * 8, &p));
    sp.wchi2 = (const double *)p;
    sp.aos2v = aos2v;
    // with K in one panel the residues of P stay for every r1 tile (and, in a scan, for
    // every set); with several panels each tile forms them again
    sp.ax_whole = sp.k_panel >= R.n2;
    if (R.mol_tag && E->tag_x == R.mol_tag && E->tag_x_buf == sp.ax.p)
        return CUTC_OK;  // the same molecule's scales (and residues) are already there
    CUTC_TRY(weighted_aos(st, R.n2, R.nA, wr2, aos2v, (int64_t)R.n2, (double *)p));
    SrcSym src{sp.wchi2, aos2v, (int64_t)R.n2, (int64_t)R.n2, sp.pairs_sym};
    CUTC_TRY(row_scales(st, src, np, (int64_t)R.n2, n_mod, sp.sc_ax, (int *)nullptr));
    if (sp.ax_whole)
        CUTC_TRY(residue_rows(st, n_mod, src, 0, np, 0, R.n2, residue_pitch(R.n2), sp.sc_ax, sp.ax.p));
    E->tag_x = R.mol_tag;
    E->tag_x_buf = sp.ax.p;
    return CUTC_OK;
}

int split_x_tile(Engine *E, const Request &R, cudaStream_t st, SplitPlan &sp, const float2 *G,
                 int nb, double *Xb, int blk_rows, int ib, cudaEvent_t gemm_begin,
                 cudaEvent_t gemm_end)
{
    const int n_mod = split_moduli(sp.n_slices);
    const int64_t np = n_pairs(R.nA);
    SrcSym sa{sp.wchi2, sp.aos2v, (int64_t)R.n2, (int64_t)R.n2, sp.pairs_sym};
    SrcDenseDF sb{G, (int64_t)R.n2};
    CUTC_TRY(row_scales(st, sb, 4 * nb, (int64_t)R.n2, n_mod, sp.sc_bx, (int *)nullptr));
    if (gemm_begin)
        CUTC_CUDA_TRY(cudaEventRecord(gemm_begin, st));
    // column (c, i) of the tile -> column c blk_rows + ib + i of the block
    const ModularOut out{Xb, np, nb, blk_rows, ib, 1.0, 0.0};
    CUTC_TRY(modular_contract(
        st, E->ws, sp.slot0 + SS_BX, sp.slot0 + SS_RES, x_residue_bytes(sp.n1t, R.n2), n_mod,
        (int)np, 4 * nb, R.n2, sp.k_panel, sp.ax, sp.ax_whole, false, sp.sc_ax, sp.sc_bx, out, sp.err, nullptr,
        [&](int64_t k0, int64_t kp, const ResiduePlanes &a) {
            return residue_rows(st, n_mod, sa, 0, (int)np, k0, kp, a.pitch, sp.sc_ax, a.p);
        },
        [&](int n0, int nc, int64_t k0, int64_t kp, const ResiduePlanes &b) {
            return residue_rows(st, n_mod, sb, n0, nc, k0, kp, b.pitch, sp.sc_bx, b.p);
        }));
    if (gemm_end)
        CUTC_CUDA_TRY(cudaEventRecord(gemm_end, st));
    return CUTC_OK;
}

int split_int2e_tile(Engine *E, const Request &R, cudaStream_t st, SplitPlan &sp,
                     const double *wr1, const double *aos1, int64_t ld1, int nb, const double *Xt,
                     double *H, double *N, bool first)
{
    Workspace &W = E->ws;
    const int slot0 = sp.slot0;
    const int nA = R.nA;
    const int np = (int)n_pairs(nA), nl = (int)n_strict_pairs(nA);
    const int n_mod = split_moduli(sp.n_slices);
    const int64_t k3 = 3 * (int64_t)nb;
    const int64_t pan_h = int2e_panel_k(n_mod, nb, np, R.k_split);
    const int64_t pan_n = int2e_panel_k(n_mod, k3, np, R.k_split);
    void *p;
    CUTC_TRY(W.get(slot0 + SS_WCHI1, std::max<size_t>(1, (size_t)nA * nb) * 8, &p));
    double *wchi = (double *)p;
    int *sc_a, *sc_h, *sc_n;
    CUTC_TRY(scale_slot(W, slot0 + SS_AI_SC, np, &sc_a));
    CUTC_TRY(scale_slot(W, slot0 + SS_BH_SC, np, &sc_h));
    CUTC_TRY(scale_slot(W, slot0 + SS_BN_SC, nl, &sc_n));
    CUTC_TRY(W.get(slot0 + SS_AI, std::max(residue_bytes(n_mod, np, pan_h),
                                           residue_bytes(n_mod, np, pan_n)), &p));
    ResiduePlanes a;
    a.p = p;
    // With the whole r1 grid in one block the B operands depend on the molecule only,
    // and a build with the same molecule tag keeps them.
    const bool whole = modular_whole(n_mod, np, nb, pan_h, kInt2eResidueBytes) &&
                       modular_whole(n_mod, nl, k3, pan_n, kInt2eResidueBytes) &&
                       modular_pass_cols(n_mod, np, np) >= np;
    const bool keep_b = whole && nb == R.n1 && R.mol_tag && E->tag_i == R.mol_tag &&
                        E->tag_i_buf == sc_h;
    SrcSym s0{wchi, aos1, (int64_t)nb, ld1, sp.pairs_sym};
    SrcAnti sn{wchi, aos1, nb, nA, ld1, sp.pairs_anti};
    if (!keep_b) {
        CUTC_TRY(weighted_aos(st, nb, nA, wr1, aos1, ld1, wchi));
        CUTC_TRY(row_scales(st, s0, np, (int64_t)nb, n_mod, sc_h, (int *)nullptr));
        CUTC_TRY(row_scales(st, sn, nl, k3, n_mod, sc_n, (int *)nullptr));
    }
    const double beta = first ? 0.0 : 1.0;
    // Xt[(m nb + i) np + p]: X_3 is column block 3, X_012 the blocks 0..2
    const double *x3 = Xt + 3 * (int64_t)nb * np;
    CUTC_TRY(row_scales_cols(st, x3, np, np, nb, n_mod, sc_a, nullptr));
    CUTC_TRY(modular_contract(
        st, W, slot0 + SS_BH, slot0 + SS_RES, kInt2eResidueBytes, n_mod, np, np, nb, pan_h, a, false, keep_b, sc_a,
        sc_h, ModularOut{H, np, np, 0, 0, 1.0, beta}, sp.err, nullptr,
        [&](int64_t k0, int64_t kp, const ResiduePlanes &o) {
            return residue_cols(st, n_mod, x3, np, np, k0, kp, o.pitch, sc_a, o.p);
        },
        [&](int n0, int nc, int64_t k0, int64_t kp, const ResiduePlanes &o) {
            return residue_rows(st, n_mod, s0, n0, nc, k0, kp, o.pitch, sc_h, o.p);
        }));
    if (nl > 0) {
        CUTC_TRY(row_scales_cols(st, Xt, np, np, k3, n_mod, sc_a, nullptr));
        CUTC_TRY(modular_contract(
            st, W, slot0 + SS_BN, slot0 + SS_RES, kInt2eResidueBytes, n_mod, np, nl, k3, pan_n, a, false, keep_b, sc_a,
            sc_n, ModularOut{N, np, nl, 0, 0, -0.5, beta}, sp.err, nullptr,
            [&](int64_t k0, int64_t kp, const ResiduePlanes &o) {
                return residue_cols(st, n_mod, Xt, np, np, k0, kp, o.pitch, sc_a, o.p);
            },
            [&](int n0, int nc, int64_t k0, int64_t kp, const ResiduePlanes &o) {
                return residue_rows(st, n_mod, sn, n0, nc, k0, kp, o.pitch, sc_n, o.p);
            }));
    }
    E->tag_i = whole && nb == R.n1 ? R.mol_tag : 0;
    E->tag_i_buf = sc_h;
    return CUTC_OK;
}

// ---- pair terms on the tensor cores -------------------------------------------------

constexpr int kPairTcMaxNuc = 20;  // K = 4 n_nuc <= 80 keeps diagonals 0..2 exact

// Slices of the pair contraction's operands: 5 (representation error 2^-45, under the
// error of a 5-slice build's contractions), or 6 for builds of 6 and 7 slices, whose
// contractions reach FP64-class errors (2^-54, below the double-float epilogue).
static int pair_tc_slices(const Request &R) { return R.n_slices >= 6 ? 6 : 5; }

bool split_pair_tc_ok(const Request &R, const int *exps, int n_terms)
{
    return R.precision == CUTC_SPLIT_BF16 && !R.pair_fp64 && R.nN <= kPairTcMaxNuc &&
           pair_df_sparse(exps, n_terms) && !getenv("CUTC_PAIR_DF") && !getenv("CUTC_PAIR_DENSE");
}

size_t split_pair_fixed_bytes(const Request &R)
{
    const int64_t K = 4 * (int64_t)R.nN;
    return (size_t)R.n2 * K * 8 +
           2 * (size_t)pair_tc_slices(R) * round_up(R.n2, kBM) * round_up(K, kBK);
}

size_t split_pair_row_bytes(const Request &R)
{
    const int64_t K = 4 * (int64_t)R.nN;
    return 16 * (size_t)K * 8 + 2 * (size_t)pair_tc_slices(R) * 16 * round_up(K, kBK) + 3 * 8 +
           16 * 4 + 64;
}

int split_pair_prepare(Engine *E, const Request &R, cudaStream_t st, const double *f2,
                       int64_t n1t, SplitPlan &sp)
{
    Workspace &W = E->ws;
    const int slot0 = sp.slot0;
    const int64_t K = 4 * (int64_t)R.nN;
    void *p;
    CUTC_TRY(W.get(slot0 + SS_F64, (size_t)R.n2 * K * 8, &p));
    sp.Fd = (double *)p;
    CUTC_TRY(W.get(slot0 + SS_C64, (size_t)16 * n1t * K * 8, &p));
    sp.Cd = (double *)p;
    CUTC_TRY(W.get(slot0 + SS_R1D, (size_t)3 * n1t * sizeof(float2), &p));
    sp.r1d = (float2 *)p;
    CUTC_TRY(W.get(slot0 + SS_BSCALE, (size_t)round_up(16 * n1t, kPairBN) * 4, &p));
    sp.bscale = (float *)p;
    const int ps = pair_tc_slices(R);
    CUTC_TRY(alloc_operand(W, slot0 + SS_AF, ps, R.n2, kBM, K, sp.AF));
    CUTC_TRY(alloc_operand(W, slot0 + SS_BC, ps, (int)(16 * n1t), kPairBN, K, sp.BC));
    CUTC_TRY(launch_pair_tc_f(st, R.n2, R.nN, f2, sp.Fd));
    note_launches(1);
    SrcDense src{sp.Fd, K};
    if (ps == 6)
        CUTC_TRY((slice_rows<6, SrcDense>(st, src, sp.AF)));
    else
        CUTC_TRY((slice_rows<5, SrcDense>(st, src, sp.AF)));
    sp.pair_slices = ps;
    sp.pair_tc = true;
    return CUTC_OK;
}

template <int S, int KB>
static int launch_pair_tc_kernel(cudaStream_t st, const CUtensorMap &ta, const CUtensorMap &tb,
                                 PairTcParams Q, int n_sm)
{
    using Cfg = PairTcCfg<S, KB>;
    static std::atomic<unsigned long long> attr_done{0};
    const unsigned long long bit = current_device_bit();
    if (!(attr_done.load() & bit)) {
        CUTC_CUDA_TRY(cudaFuncSetAttribute(pair_tc_kernel<S, KB>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem));
        attr_done.fetch_or(bit);
    }
    // about eight CTAs per SM, each walking a run of N tiles with its F tile resident
    const int64_t want = 8 * (int64_t)n_sm;
    const int64_t chunks = std::max<int64_t>(
        1, std::min<int64_t>(Q.tiles_n, (want + Q.tiles_m - 1) / Q.tiles_m));
    Q.chunk = (int)((Q.tiles_n + chunks - 1) / chunks);
    const int64_t grid = (int64_t)Q.tiles_m * ((Q.tiles_n + Q.chunk - 1) / Q.chunk);
    if (grid > INT32_MAX) {
        cutc_set_error(CUTC_ERR_INVALID, "pair grid of %lld CTAs", (long long)grid);
        return CUTC_ERR_INVALID;
    }
    pair_tc_kernel<S, KB><<<(unsigned)grid, Cfg::kThreads, Cfg::kSmem, st>>>(ta, tb, Q);
    CUTC_CUDA_TRY(cudaGetLastError());
    return CUTC_OK;
}

template <int S>
static int pair_tile(Engine *E, cudaStream_t st, SplitPlan &sp, const PairDfArgs &P,
                     const double *rn, double a_en)
{
    constexpr int BN = kPairBN;
    const int64_t K = 4 * (int64_t)P.nN;
    CUTC_TRY(launch_pair_tc_coef(st, P.i0, P.n1b, P.nN, P.r1, rn, a_en, P.coef, P.exps,
                                 P.term_off, sp.Cd, sp.r1d));
    Operand B = sp.BC;
    B.M = 16 * P.n1b;
    B.Mpad = (int)round_up(B.M, BN);
    SrcDense src{sp.Cd, K};
    CUTC_TRY((slice_rows<S, SrcDense>(st, src, B)));
    exp_scale_kernel<<<ceil_div(B.Mpad, 256), 256, 0, st>>>(B.ex, B.Mpad, sp.bscale);
    CUTC_CUDA_TRY(cudaGetLastError());
    CUtensorMap ta, tb;
    CUTC_TRY(make_tmap(&ta, sp.AF.sl, (int64_t)S * sp.AF.Mpad, sp.AF.Kpad, kBM));
    CUTC_TRY(make_tmap(&tb, B.sl, (int64_t)S * B.Mpad, B.Kpad, BN));
    PairTcParams Q;
    Q.tiles_m = sp.AF.Mpad / kBM;
    Q.tiles_n = B.Mpad / BN;
    Q.chunk = 1;
    Q.Mpad = sp.AF.Mpad;
    Q.Npad = B.Mpad;
    Q.ea = sp.AF.ex;
    Q.bscale = sp.bscale;
    Q.r1d = sp.r1d;
    Q.P = P;
    Q.err = sp.err;
    const int KB = (int)(sp.AF.Kpad / kBK);
    switch (KB) {
    case 1: CUTC_TRY((launch_pair_tc_kernel<S, 1>(st, ta, tb, Q, E->n_sm))); break;
    case 2: CUTC_TRY((launch_pair_tc_kernel<S, 2>(st, ta, tb, Q, E->n_sm))); break;
    case 3: CUTC_TRY((launch_pair_tc_kernel<S, 3>(st, ta, tb, Q, E->n_sm))); break;
    default:
        cutc_set_error(CUTC_ERR_INVALID, "pair contraction of K = %lld", (long long)K);
        return CUTC_ERR_INVALID;
    }
    note_launches(3);
    return CUTC_OK;
}

int split_pair_tile(Engine *E, const Request &R, cudaStream_t st, SplitPlan &sp,
                    const PairDfArgs &P, const double *rn, double a_en)
{
    (void)R;
    if (P.n1b <= 0 || P.n2 <= 0)
        return CUTC_OK;
    return sp.pair_slices == 6 ? pair_tile<6>(E, st, sp, P, rn, a_en)
                               : pair_tile<5>(E, st, sp, P, rn, a_en);
}

// One CTA waits on a pipeline barrier that nothing completes, with the bounded wait
// the tensor-core kernels use; it records whether the wait gave up (2) or, against
// all expectation, completed (1).
__global__ void wait_limit_kernel(int *result)
{
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        tc::mbar_init(tc::smem_u32(&bar), 1);
        tc::fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0)
        *result = tc::mbar_wait(tc::smem_u32(&bar), 0, nullptr) ? 1 : 2;
}

int split_wait_limit_check(Engine *E)
{
    void *p;
    CUTC_TRY(E->ws.get(240, 64, &p));
    int *d = (int *)p;
    CUTC_CUDA_TRY(cudaMemsetAsync(d, 0, 4, E->stream));
    wait_limit_kernel<<<1, 32, 0, E->stream>>>(d);
    CUTC_CUDA_TRY(cudaGetLastError());
    int h = 0;
    CUTC_CUDA_TRY(cudaMemcpyAsync(&h, d, 4, cudaMemcpyDeviceToHost, E->stream));
    CUTC_CUDA_TRY(cudaStreamSynchronize(E->stream));
    if (h == 2) {
        cutc_set_error(CUTC_ERR_TIMEOUT, "a pipeline wait gave up after its limit (as checked)");
        return CUTC_ERR_TIMEOUT;
    }
    cutc_set_error(CUTC_ERR_CUDA, "the wait-limit check's barrier completed (result %d)", h);
    return CUTC_ERR_CUDA;
}

int split_check(cudaStream_t st, SplitPlan &sp)
{
    int herr = 0;
    CUTC_CUDA_TRY(cudaMemcpyAsync(&herr, sp.err, 4, cudaMemcpyDeviceToHost, st));
    CUTC_CUDA_TRY(cudaStreamSynchronize(st));
    if (herr) {
        cutc_set_error(CUTC_ERR_TIMEOUT, "a tensor-core pipeline wait gave up (code %d)", herr);
        return CUTC_ERR_TIMEOUT;
    }
    return CUTC_OK;
}

// C = alpha A B^T of two sources through the split form, synchronous on st.
template <class Src>
static int gemm_sources(Engine *E, cudaStream_t st, int base, int n_slices, int M, int N,
                        int64_t K, Src sa, Src sb, double alpha, double *C, int64_t ldc)
{
    Workspace &W = E->ws;
    const int n_mod = split_moduli(n_slices);
    const int64_t pan = panel_k(K, M, 0);
    int *sc_a, *sc_b;
    void *p;
    CUTC_TRY(scale_slot(W, base, M, &sc_a));
    CUTC_TRY(scale_slot(W, base + 1, N, &sc_b));
    CUTC_TRY(W.get(base + 2, 64, &p));
    int *err = (int *)p;
    CUTC_TRY(W.get(base + 3, residue_bytes(n_mod, M, pan), &p));
    ResiduePlanes a;
    a.p = p;
    CUTC_CUDA_TRY(cudaMemsetAsync(err, 0, 4, st));
    CUTC_TRY(row_scales(st, sa, M, K, n_mod, sc_a, (int *)nullptr));
    CUTC_TRY(row_scales(st, sb, N, K, n_mod, sc_b, (int *)nullptr));
    CUTC_TRY(modular_contract(
        st, W, base + 4, base + 5, (size_t)8 << 30, n_mod, M, N, K, pan, a, false, false, sc_a, sc_b,
        ModularOut{C, ldc, N, 0, 0, alpha, 0.0}, err, nullptr,
        [&](int64_t k0, int64_t kp, const ResiduePlanes &o) {
            return residue_rows(st, n_mod, sa, 0, M, k0, kp, o.pitch, sc_a, o.p);
        },
        [&](int n0, int nc, int64_t k0, int64_t kp, const ResiduePlanes &o) {
            return residue_rows(st, n_mod, sb, n0, nc, k0, kp, o.pitch, sc_b, o.p);
        }));
    SplitPlan sp;
    sp.err = err;
    return split_check(st, sp);
}

// Split-precision GEMM on device arrays: C[m + ldc n] = sum_k A[m K + k] B[n K + k].
int split_gemm_dense(Engine *E, cudaStream_t st, int n_slices, int M, int N, int64_t K,
                     const double *A, const double *B, double *C, int64_t ldc)
{
    return gemm_sources(E, st, 200, n_slices, M, N, K, SrcDense{A, K}, SrcDense{B, K}, 1.0, C, ldc);
}

// C[m + ldc n] = alpha sum_k [A1 | A2][m, k] [B1 | B2][n, k] through the split form: the
// two products of the same output as ONE contraction over K1 + K2 (one row scale per row
// of the concatenation).  A1, B1 are K1-contiguous, A2, B2 K2-contiguous (device arrays);
// synchronous on st.
int split_gemm_concat(Engine *E, cudaStream_t st, int n_slices, int M, int N, int64_t K1,
                      const double *A1, const double *B1, int64_t K2, const double *A2,
                      const double *B2, double alpha, double *C, int64_t ldc)
{
    return gemm_sources(E, st, 210, n_slices, M, N, K1 + K2, SrcConcat{A1, A2, K1, K2},
                        SrcConcat{B1, B2, K1, K2}, alpha, C, ldc);
}

}  // namespace cutc
