// Modular contraction: residue products on tcgen05 CTA pairs, and the FP64 results from
// their residues (moduli.cuh has the arithmetic).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>

#include "modular.cuh"
#include "tc.cuh"

namespace cutc {

// ---------------------------------------------------------------------------
// the residue products
// ---------------------------------------------------------------------------

// One CTA pair (a cluster of two) computes a 256 x BN tile of one modulus: the pair's
// tcgen05.mma (cta_group::2, M = 256) takes 128 rows of A and half of B's rows from each
// CTA's shared memory.  Against one CTA with a 128 x 256 tile this reads 8 instead of
// 12 KB from L2 per 16-wide K step and SM, 64 B per clock at the tensor pipe's full rate.
// Bound by the tensor pipe, the accumulators' reads beside it, and in long runs the power
// cap: M 7260, N 16384, K 16384 with 11 moduli takes 23.6 ms, 1817 TF/s of BF16 products
// (cuBLAS: 1898 in a burst, 1704 sustained).  The 5-slice kernel that this replaces, with
// a 128 x 48 tile of five stacked accumulators, ran 15 products at 1551 TF/s.  The medium
// build (n_ao 120, 25k x 80k, 13 moduli): 1361 -> 1110 ms, with smaller errors (int_2e
// 1.7e-12 -> 1e-13).
constexpr int kTileM = 256, kBK = 64;     // 64 BF16 = 128-byte rows (128B swizzle)
constexpr int kChunkBlocks = 8;           // 512 K: sums of products of residues below 2^24
constexpr int kEpiWarps = 16;             // 4 lane quarters x 4 column groups
constexpr int kTmaWarp = kEpiWarps, kMmaWarp = kEpiWarps + 1;
constexpr int kGemmThreads = (kEpiWarps + 2) * 32;
constexpr int kGroupN = 8;                // column tiles per raster group
constexpr int kResidentBlocks = 128;      // K blocks up to which pairs stay resident (8192 K)

template <int BN>
struct ModCfg {
    static constexpr int kA = 128 * kBK * 2;
    static constexpr int kB = BN / 2 * kBK * 2;
    static constexpr int kStage = kA + kB;
    static constexpr int kStages = 6;
    static constexpr int kSmem = kStages * kStage + 1024 + 256;
    static constexpr uint32_t kTmemCols = 2 * BN;  // two accumulator buffers (a power of two)
    static constexpr int kCols = BN / 4;           // columns per epilogue warp
    static_assert(kCols % 16 == 0, "16 columns per tensor-memory load");
    static_assert(kSmem <= 227 * 1024, "shared memory");
    static_assert(kTmemCols <= 512, "tensor memory");
};

// A residue r of a result is stored as the low half of the bits of the float r + kResidueBias,
// whose high half is kResidueHigh.
constexpr float kResidueBias = 12582912.0f + (float)kResidueOffset;  // 1.5 * 2^23 + 2^9
constexpr unsigned kResidueHigh = 0x4b40u;

struct ModGemmParams {
    int planes, M, N, tiles_m, tiles_n;
    int magnitudes;            // the plane of magnitudes' sums, if any
    int nkb;                   // K blocks of the panel
    int accumulate;            // add to the residues in out
    unsigned short *out;       // out[i plane + n ldm + m]
    int64_t ldm, plane;
    float p[moduli::kMax + 1], inv[moduli::kMax + 1];  // 0: sums, not residues
    int *err;                  // set to a non-zero code if a bounded wait gave up
};

// The bits of a plane's entry: of a sum of magnitudes, zero stays zero and others are
// 1 .. kMagnitudeCap; a residue is itself (the bounds are beyond it).
__device__ __forceinline__ uint32_t bounded_sum(float x, bool sum)
{
    return __float_as_uint(x == 0.0f ? x : fminf(fmaxf(x, sum ? 1.0f : -1024.0f), (float)kMagnitudeCap));
}

// kResident: the pair walks tasks of its own, a grid's width apart; else it has one.  kMag:
// plane P.magnitudes holds sums.
template <int BN, bool kResident, bool kMag>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
modular_gemm_kernel(const __grid_constant__ CUtensorMap tmA,
                    const __grid_constant__ CUtensorMap tmB, const __grid_constant__ ModGemmParams P)
{
    using Cfg = ModCfg<BN>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // (the dynamic shared memory starts at the same offset in both CTAs)
    const uint32_t pad = (1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u;
    uint8_t *smem = smem_raw + pad;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + Cfg::kStages * Cfg::kStage);
    uint64_t *full = bars;                       // leader: both CTAs' copies of a stage landed
    uint64_t *empty = bars + Cfg::kStages;       // each: the MMAs have read the stage
    uint64_t *tfull = bars + 2 * Cfg::kStages;   // each: the accumulators hold a chunk
    uint64_t *tempty = tfull + 2;                // leader: both CTAs' epilogues have read them
    uint64_t *drain = tempty + 2;
    uint64_t *gone = drain + 1;                  // each: the other has given its tensor memory back
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(gone + 1);
    volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = tc::cluster_rank();
    const bool leader = rank == 0;

    // Tasks (one tile of one modulus each), every pair walking its share (one task, or the
    // epilogue of a task beside the MMAs of the next).  Moduli outermost, then a grouped raster
    // (kGroupN column tiles sweep the row tiles, so concurrent pairs share their tiles of
    // A and B through L2).
    const int per_mod = P.tiles_m * P.tiles_n;
    const int n_tasks = P.planes * per_mod, first = (int)(blockIdx.x >> 1);
    const int stride = (int)(gridDim.x >> 1);
    struct Tile {
        int z, m0, n0;
    };
    auto tile = [&](int task) {
        Tile o;
        o.z = task / per_mod;
        const int t = task % per_mod;
        const int per_group = kGroupN * P.tiles_m;
        const int gfirst = (t / per_group) * kGroupN;
        const int gsize = min(P.tiles_n - gfirst, kGroupN);
        o.n0 = (gfirst + (t % per_group) % gsize) * BN;
        o.m0 = ((t % per_group) / gsize) * kTileM + (int)rank * 128;
        return o;
    };
    const int nkb = P.nkb;

    if (threadIdx.x == 0) {
        for (int i = 0; i < Cfg::kStages; i++) {
            tc::mbar_init(tc::smem_u32(&full[i]), 1);
            tc::mbar_init(tc::smem_u32(&empty[i]), 1);
        }
        for (int i = 0; i < 2; i++) {
            tc::mbar_init(tc::smem_u32(&tfull[i]), 1);
            tc::mbar_init(tc::smem_u32(&tempty[i]), 2 * kEpiWarps);
        }
        tc::mbar_init(tc::smem_u32(drain), 1);
        tc::mbar_init(tc::smem_u32(gone), 1);
        *s_abort = 0;
        tc::fence_mbar_init();
    }
    // A pair's allocation takes both CTAs: neither asks before the other has started, nor
    // leaves (below) before the other has given its part back.  Without this, with kernels of
    // other streams on the device, an allocation could wait for good.
    tc::cluster_sync();
    if (warp == kMmaWarp) {
        tc::tmem_alloc_pair(tc::smem_u32(s_tmem), Cfg::kTmemCols);
        tc::tmem_relinquish_pair();
    }
    if (warp == kTmaWarp && lane == 0) {
        tc::tma_prefetch(&tmA);
        tc::tma_prefetch(&tmB);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync();  // both CTAs' barriers are initialised
    tc::fence_after_sync();
    const uint32_t tbase = *s_tmem;

    auto fail = [&](int code) {
        *s_abort = 1;
        atomicExch(P.err, code);
    };

    // A stage's barriers complete once per round; `phase` is the parity of the current one
    // (a wait for the round before the first returns at once).
    if (warp == kTmaWarp) {
        if (lane == 0) {
            uint32_t stage = 0, phase = 0, issued = 0;
            bool ok = true;
            for (int task = first; task < n_tasks && ok; task = kResident ? task + stride : n_tasks) {
                const Tile o = tile(task);
                const int nb = o.n0 + (int)rank * (BN / 2);
                for (int kb = 0; kb < nkb; kb++) {
                    if (!tc::mbar_wait(tc::smem_u32(&empty[stage]), phase ^ 1, s_abort)) {
                        fail(21);
                        ok = false;
                        break;
                    }
                    const uint32_t fb = tc::smem_u32(&full[stage]);
                    if (leader)
                        tc::mbar_arrive_expect_tx(fb, 2 * Cfg::kStage);
                    const uint32_t fl = tc::map_to_rank(fb, 0);
                    const uint32_t st = tc::smem_u32(smem) + stage * Cfg::kStage;
                    tc::tma_load_3d_pair(st, &tmA, kb * kBK, o.m0, o.z, fl);
                    tc::tma_load_3d_pair(st + Cfg::kA, &tmB, kb * kBK, nb, o.z, fl);
                    issued++;
                    if (++stage == Cfg::kStages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            // the last MMAs have read their stages, and signalled so, before this CTA goes away
            for (uint32_t i = 0, t = stage, ph = phase ^ 1; i < (uint32_t)Cfg::kStages && ok; i++) {
                if (!tc::mbar_wait(tc::smem_u32(&empty[t]), ph, s_abort)) {
                    fail(26);
                    ok = false;
                }
                if (++t == Cfg::kStages) {
                    t = 0;
                    ph ^= 1;
                }
            }
            if (*s_abort && leader) {
                // let the copies already issued land before the pair goes away
                for (uint32_t i = 0; i < min(issued, (uint32_t)Cfg::kStages); i++) {
                    if (stage-- == 0) {
                        stage = Cfg::kStages - 1;
                        phase ^= 1;
                    }
                    tc::mbar_wait(tc::smem_u32(&full[stage]), phase, nullptr);
                }
            }
        }
    } else if (warp == kMmaWarp) {
        if (leader && lane == 0) {
            bool ok = true;
            const uint32_t idesc = tc::idesc_bf16_f32(kTileM, BN);
            const uint64_t ad0 = tc::smem_desc_sw128(tc::smem_u32(smem));
            const uint64_t bd0 = tc::smem_desc_sw128(tc::smem_u32(smem) + Cfg::kA);
            uint32_t stage = 0, phase = 0, buf = 0, bphase = 0;
            for (int task = first; task < n_tasks && ok; task = kResident ? task + stride : n_tasks) {
                for (int kb0 = 0; kb0 < nkb && ok; kb0 += kChunkBlocks) {
                    if (!tc::mbar_wait(tc::smem_u32(&tempty[buf]), bphase ^ 1, s_abort)) {
                        fail(22);
                        ok = false;
                        break;
                    }
                    tc::fence_after_sync();
                    const int kb1 = min(nkb, kb0 + kChunkBlocks);
                    for (int kb = kb0; kb < kb1; kb++) {
                        if (!tc::mbar_wait(tc::smem_u32(&full[stage]), phase, s_abort)) {
                            fail(23);
                            ok = false;
                            break;
                        }
                        tc::fence_after_sync();
                        const uint64_t ad = ad0 + stage * (Cfg::kStage >> 4);
                        const uint64_t bd = bd0 + stage * (Cfg::kStage >> 4);
#pragma unroll
                        for (int k16 = 0; k16 < kBK / 16; k16++)  // 32 bytes further in each row
                            tc::mma_bf16_pair(tbase + BN * buf, ad + 2 * k16, bd + 2 * k16, idesc,
                                              kb > kb0 || k16 > 0);
                        tc::mma_commit_pair(tc::smem_u32(&empty[stage]));
                        if (++stage == Cfg::kStages) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                    if (ok)
                        tc::mma_commit_pair(tc::smem_u32(&tfull[buf]));
                    bphase ^= buf;
                    buf ^= 1;
                }
            }
            // (without a failure the copying warps wait for the last MMAs)
            if (!ok) {
                tc::mma_commit_pair(tc::smem_u32(drain));
                if (!tc::mbar_wait(tc::smem_u32(drain), 0, nullptr))
                    fail(25);
            }
        }
    } else {
        // ---- epilogue: running residues of the warp's 32 rows x kCols columns ----------
        constexpr int CP = Cfg::kCols / 2;  // column pairs (one f32x2 each)
        const int q = warp & 3, grp = warp >> 2;
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        const uint32_t coff = (uint32_t)(grp * Cfg::kCols);
        const uint64_t magic = tc::f2_dup(12582912.0f);  // 1.5 * 2^23
        const uint64_t bias = tc::f2_dup(kResidueBias);
        const uint32_t te0 = tc::map_to_rank(tc::smem_u32(&tempty[0]), 0);
        const uint32_t te1 = tc::map_to_rank(tc::smem_u32(&tempty[1]), 0);
        bool ok = true;
        uint32_t buf = 0, bphase = 0;
        for (int task = first; task < n_tasks && ok; task = kResident ? task + stride : n_tasks) {
            const Tile o = tile(task);
            const int m = o.m0 + q * 32 + lane;
            unsigned short *dst = P.out + o.z * P.plane + (int64_t)(o.n0 + (int)coff) * P.ldm + m;
            const int ncol = P.N - o.n0 - (int)coff;  // columns of this warp that exist
            const uint64_t inv = tc::f2_dup(P.inv[o.z]), negp = tc::f2_dup(-P.p[o.z]);
            uint64_t acc[CP];
#pragma unroll
            for (int j = 0; j < CP; j++)
                acc[j] = 0ull;
            if (P.accumulate && m < P.M) {
#pragma unroll
                for (int j = 0; j < CP; j++) {
                    const unsigned a = 2 * j < ncol ? dst[(int64_t)(2 * j) * P.ldm] : 512u;
                    const unsigned b = 2 * j + 1 < ncol ? dst[(int64_t)(2 * j + 1) * P.ldm] : 512u;
                    acc[j] = tc::f2_sub(tc::f2_pack((kResidueHigh << 16) | a, (kResidueHigh << 16) | b),
                                        bias);
                }
            }
            for (int kb0 = 0; kb0 < nkb; kb0 += kChunkBlocks) {
                if (!tc::mbar_wait(tc::smem_u32(&tfull[buf]), bphase, s_abort)) {
                    fail(24);
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
                // acc <- (acc + v) mod p: |v| + |acc| < 2^24, every step exact
#pragma unroll
                for (int h = 0; h < Cfg::kCols / 16; h++) {
                    float v[16];
                    tc::tmem_ld16(tbase + lane_off + BN * buf + coff + 16u * h, v);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        uint64_t &a = acc[8 * h + j];
                        const uint64_t s =
                            tc::f2_add(a, tc::f2_pack(__float_as_uint(v[2 * j]),
                                                      __float_as_uint(v[2 * j + 1])));
                        const uint64_t d = tc::f2_sub(tc::f2_fma(s, inv, magic), magic);
                        a = tc::f2_fma(d, negp, s);
                    }
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0)
                    tc::mbar_arrive_cluster(buf ? te1 : te0);
                bphase ^= buf;
                buf ^= 1;
            }
            if (ok && m < P.M) {
#pragma unroll
                for (int j = 0; j < CP; j++) {
                    uint64_t w = acc[j];
                    if constexpr (kMag)
                        w = tc::f2_pack(bounded_sum(tc::f2_lo(w), o.z == P.magnitudes),
                                        bounded_sum(tc::f2_hi(w), o.z == P.magnitudes));
                    w = tc::f2_add(w, bias);
                    if (2 * j < ncol)
                        dst[(int64_t)(2 * j) * P.ldm] = (unsigned short)w;
                    if (2 * j + 1 < ncol)
                        dst[(int64_t)(2 * j + 1) * P.ldm] = (unsigned short)(w >> 32);
                }
            }
        }
    }

    __syncwarp();
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync();  // neither CTA leaves while the other may signal it or read its operands
    tc::fence_after_sync();
    if (warp == kMmaWarp) {
        tc::tmem_dealloc_pair(tbase, Cfg::kTmemCols);
        __syncwarp();
        if (lane == 0) {  // (the other waits for this arrival before it goes away)
            tc::mbar_arrive_cluster(tc::map_to_rank(tc::smem_u32(gone), rank ^ 1));
            if (!tc::mbar_wait(tc::smem_u32(gone), 0, nullptr))
                fail(27);
        }
    }
}

// ---------------------------------------------------------------------------
// the results
// ---------------------------------------------------------------------------

struct CombineParams {
    int M, ncols, n0;
    const unsigned short *res;
    int64_t ldm, plane;
    const int *sa, *sb;
    ModularOut out;
    int alpha_exp, alpha_neg, alpha_mul, beta_mode;  // beta_mode: 0, 1 or 2 (any other beta)
    const int *err;
    LeftResults *left;
};

// Tables of the Chinese remainder theorem for N moduli: V = sum_i r_i W_i mod M with
// W_i = (M / p_i) ((M / p_i)^-1 mod p_i), in 12-bit limbs (FP32 pairs, both lanes the same
// value) and as fractions W_i / M.
constexpr int kLimbBits = 12;
constexpr int crt_limbs(int n)
{
    return n <= 8 ? 6 : n <= 9 ? 7 : n <= 11 ? 8 : n <= 12 ? 9 : n <= 13 ? 10 : n <= 15 ? 11 : 12;
}

template <int N>
struct CrtTab {
    static constexpr int L = crt_limbs(N);
    uint64_t w[N][L], frac[N];
};

// An unsigned integer of W 64-bit words.
template <int W>
struct Words {
    unsigned long long w[W];
    constexpr Words times(unsigned m) const
    {
        Words r{};
        unsigned __int128 c = 0;
        for (int i = 0; i < W; i++) {
            c += (unsigned __int128)w[i] * m;
            r.w[i] = (unsigned long long)c;
            c >>= 64;
        }
        return r;
    }
    constexpr Words over(unsigned d, unsigned *rest) const
    {
        Words r{};
        unsigned __int128 c = 0;
        for (int i = W - 1; i >= 0; i--) {
            c = (c << 64) | w[i];
            r.w[i] = (unsigned long long)(c / d);
            c %= d;
        }
        *rest = (unsigned)c;
        return r;
    }
    constexpr unsigned bits12(int b) const
    {
        const int i = b / 64, s = b % 64;
        unsigned long long v = i < W ? w[i] >> s : 0;
        if (s > 52 && i + 1 < W)
            v |= w[i + 1] << (64 - s);
        return (unsigned)v & 0xfffu;
    }
    constexpr double value() const
    {
        double r = 0.0;
        for (int i = W - 1; i >= 0; i--)
            r = r * 18446744073709551616.0 + (double)w[i];
        return r;
    }
};

// Words that hold the results' integers: |V| < M / 2 with the sign (M < 2^126.01 of 15 moduli,
// 2^142.4 of 17).
template <int N>
constexpr int kWords = N <= 15 ? 2 : 3;

template <int N>
constexpr Words<3> modulus()
{
    Words<3> M{{1, 0, 0}};
    for (int i = 0; i < N; i++)
        M = M.times((unsigned)moduli::prime(i));
    return M;
}

constexpr uint32_t positive_code(double x)  // the bits of a positive double as a float
{
    int e = 0;
    while (x >= 2.0) {
        x *= 0.5;
        e++;
    }
    while (x < 1.0) {
        x *= 2.0;
        e--;
    }
    return ((uint32_t)(127 + e) << 23) + (uint32_t)((x - 1.0) * 8388608.0 + 0.5);
}

template <int N>
constexpr CrtTab<N> make_crt_tab()
{
    CrtTab<N> t{};
    const Words<3> M = modulus<N>();
    for (int i = 0; i < N; i++) {
        const int p = moduli::prime(i);
        unsigned rest = 0, mod = 0;
        const Words<3> q = M.over((unsigned)p, &rest);
        (void)q.over((unsigned)p, &mod);
        int inv = moduli::inverse((int)mod, p);
        if (inv < 0)
            inv += p;
        const Words<3> w = q.times((unsigned)inv);
        for (int l = 0; l < CrtTab<N>::L; l++)
            t.w[i][l] = dup_code(float_code((int)w.bits12(kLimbBits * l)));
        t.frac[i] = dup_code(positive_code(w.value() / M.value()));
    }
    return t;
}

static __constant__ const CrtTab<8> c_crt8 = make_crt_tab<8>();
static __constant__ const CrtTab<9> c_crt9 = make_crt_tab<9>();
static __constant__ const CrtTab<10> c_crt10 = make_crt_tab<10>();
static __constant__ const CrtTab<11> c_crt11 = make_crt_tab<11>();
static __constant__ const CrtTab<12> c_crt12 = make_crt_tab<12>();
static __constant__ const CrtTab<13> c_crt13 = make_crt_tab<13>();
static __constant__ const CrtTab<15> c_crt15 = make_crt_tab<15>();
static __constant__ const CrtTab<17> c_crt17 = make_crt_tab<17>();

template <int N>
__device__ __forceinline__ const CrtTab<N> &crt_tab()
{
    if constexpr (N == 8)
        return c_crt8;
    else if constexpr (N == 9)
        return c_crt9;
    else if constexpr (N == 10)
        return c_crt10;
    else if constexpr (N == 11)
        return c_crt11;
    else if constexpr (N == 12)
        return c_crt12;
    else if constexpr (N == 13)
        return c_crt13;
    else if constexpr (N == 15)
        return c_crt15;
    else
        return c_crt17;
}

// (-1)^neg a 2^k rounded to nearest even, in integer arithmetic (GB300's FP64 pipe is slow)
__device__ __forceinline__ double scaled_double(unsigned __int128 a, bool neg, int k)
{
    const unsigned long long ah = (unsigned long long)(a >> 64);
    if (a == 0)
        return 0.0;
    const int lz = ah ? __clzll((long long)ah) : 64 + __clzll((long long)(unsigned long long)a);
    a <<= lz;  // the leading bit at bit 127
    const unsigned long long h = (unsigned long long)(a >> 64), l = (unsigned long long)a;
    const int E = 1023 + 127 - lz + k;
    unsigned long long bits;
    if (E >= 1 && E <= 2046) {  // m's leading bit (or its carry) adds one to the exponent field
        unsigned long long m = h >> 11;  // 53 bits
        const unsigned rest = (unsigned)h & 0x7ffu;
        m += rest > 0x400u || (rest == 0x400u && (l != 0 || (m & 1))) ? 1 : 0;
        bits = ((unsigned long long)(E - 1) << 52) + m;
    } else if (E > 2046) {
        bits = 0x7ffull << 52;
    } else {  // subnormal: the multiple of 2^-1074 in place of the 53 bits
        const int drop = 76 - E;
        unsigned long long m = 0;
        if (drop < 128)
            m = (unsigned long long)(a >> drop);
        if (drop <= 128) {
            const unsigned __int128 rest = drop < 128 ? a << (128 - drop) : a;
            const unsigned __int128 half = (unsigned __int128)1 << 127;
            m += rest > half || (rest == half && (m & 1)) ? 1 : 0;
        }
        bits = m;
    }
    return __longlong_as_double((long long)(bits | (neg ? 1ull << 63 : 0ull)));
}

// (sum_l v[l] 2^12l - q M) 2^k as a double: v[l] integer-valued floats below 2^24 in
// magnitude; all integer arithmetic is modulo 2^128 or 2^192, which hold the difference.
template <int N>
__device__ __forceinline__ double limbs_double(const float (&v)[CrtTab<N>::L], int q, int k)
{
    constexpr int L = CrtTab<N>::L, W = kWords<N>, top = (L - 1) / 3;
    constexpr Words<3> M = modulus<N>();
    auto part = [&](int g) {  // three limbs, below 2^(24 + 24) in magnitude
        long long s = 0;
        const int n = g == top ? L - 3 * g : 3;
#pragma unroll
        for (int l = n - 1; l >= 0; l--)
            s = s * (1 << kLimbBits) + __float2int_rn(v[3 * g + l]);
        return s;
    };
    if constexpr (W == 2) {
        unsigned __int128 r = 0;
#pragma unroll
        for (int g = top; g >= 0; g--)
            r = (r << (3 * kLimbBits)) + (unsigned __int128)(__int128)part(g);
        constexpr unsigned __int128 m = ((unsigned __int128)M.w[1] << 64) | M.w[0];
        r -= (unsigned __int128)(__int128)q * m;
        const bool neg = (long long)(r >> 64) < 0;
        return scaled_double(neg ? -r : r, neg, k);
    } else {
        unsigned __int128 lo = 0;  // 192 bits: hi, lo
        unsigned long long hi = 0;
        auto add = [&](__int128 x) {  // (sign-extended)
            const unsigned __int128 s = lo + (unsigned __int128)x;
            hi += (x < 0 ? ~0ull : 0ull) + (s < lo ? 1ull : 0ull);
            lo = s;
        };
#pragma unroll
        for (int g = top; g >= 0; g--) {
            hi = (hi << 36) | (unsigned long long)(lo >> 92);
            lo <<= 36;
            add(part(g));
        }
        static_assert(3 * kLimbBits == 36, "");
        // -q M, word by word: |q| < 2^13
        add(-((__int128)q * (long long)(M.w[0] & 0xffffffffull)));
        add(-((__int128)q * (long long)(M.w[0] >> 32) * ((__int128)1 << 32)));
        constexpr unsigned long long m1 = M.w[1] & 0xffffffffull, m2 = M.w[1] >> 32;
        add(-((__int128)q * (long long)m1 * ((__int128)1 << 64)));
        // the rest from 2^96 up
        const __int128 t = -((__int128)q * (__int128)(m2 | (M.w[2] << 32)));
        const unsigned __int128 tl = (unsigned __int128)t << 96;
        const unsigned __int128 s = lo + tl;
        hi += (unsigned long long)(t >> 32) + (s < lo ? 1ull : 0ull);
        lo = s;
        const bool neg = (long long)hi < 0;
        if (neg) {
            lo = -lo;
            hi = ~hi + (lo == 0 ? 1ull : 0ull);
        }
        if (hi) {  // to 128 bits, what falls off kept as the last bit
            const int n = 64 - __clzll((long long)hi);
            const bool rest = (lo & (((unsigned __int128)1 << n) - 1)) != 0;
            lo = ((unsigned __int128)hi << (128 - n)) | (lo >> n);
            lo |= rest ? 1 : 0;
            k += n;
        }
        return scaled_double(lo, neg, k);
    }
}

// Residues -> the integer V = sum_i r_i W_i - q M (Chinese remainder theorem) -> FP64,
// rounded once.  The limbs' sums stay below 2^24 (17 residues of 181 times 12 bits), so
// their FP32 operations are exact; sum_i r_i W_i / M is off by less than 0.0025 (17 roundings
// of sums below 4096), and |V| <= 0.4935 M by the row scales (0.4914, and 0.0014 in each
// log2 norm), so q is its nearest integer.
// Consecutive threads take consecutive m, two per thread in f32x2 operations; bound by
// these N (L + 1) operations and the integer work, where Garner's mixed-radix digits took
// 5 N (N - 1) / 2.
template <int N, bool kChecked>
__global__ void __launch_bounds__(128) combine_kernel(const CombineParams P)
{
    const int m = 2 * (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (m >= P.M)
        return;
    constexpr int L = CrtTab<N>::L;
    const CrtTab<N> &tab = crt_tab<N>();
    const bool failed = *P.err != 0;
    const uint64_t magic = tc::f2_dup(12582912.0f);
    const uint64_t bias = tc::f2_dup(kResidueBias);
    const int s0 = P.sa[m], s1 = m + 1 < P.M ? P.sa[m + 1] : 0;
    for (int c = blockIdx.y; c < P.ncols; c += gridDim.y) {
        const unsigned short *src = P.res + (int64_t)c * P.ldm + m;
        unsigned word[N];
#pragma unroll
        for (int i = 0; i < N; i++)
            word[i] = *reinterpret_cast<const unsigned *>(src + i * P.plane);
        uint64_t v[L], t = 0ull;
#pragma unroll
        for (int l = 0; l < L; l++)
            v[l] = 0ull;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const uint64_t r = tc::f2_sub(tc::f2_pack(__byte_perm(word[i], kResidueHigh, 0x5410),
                                                      __byte_perm(word[i], kResidueHigh, 0x5432)),
                                          bias);
            t = tc::f2_fma(r, tab.frac[i], t);
#pragma unroll
            for (int l = 0; l < L; l++)
                v[l] = tc::f2_fma(r, tab.w[i][l], v[l]);
        }
        const uint64_t q = tc::f2_add(t, magic);  // its bits: q + those of 1.5 * 2^23
        const int sn = P.sb[c], n = P.n0 + c;
        unsigned sums = 0;
        if constexpr (kChecked)
            sums = *reinterpret_cast<const unsigned *>(src + N * P.plane);
        const int64_t col = (int64_t)(n / P.out.ncol_group) * P.out.group_stride + P.out.col0 +
                            n % P.out.ncol_group;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (m + h >= P.M)
                break;
            const int gm = P.out.row0 + m + h;
            const int64_t row = P.out.nrow_group ? (int64_t)(gm / P.out.nrow_group) * P.out.row_stride +
                                                       gm % P.out.nrow_group
                                                 : gm;
            double *dst = P.out.C + row + P.out.ldc * col;
            float f[L];
#pragma unroll
            for (int l = 0; l < L; l++)
                f[l] = h ? tc::f2_hi(v[l]) : tc::f2_lo(v[l]);
            const int sm = h ? s1 : s0;
            if (kChecked && result_left(h ? sums >> 16 : sums & 0xffffu, sm, sn)) {
                if (*(volatile int *)&P.left->count < kMaxListed) {
                    const int at = atomicAdd(&P.left->count, 1);
                    if (at < kMaxListed)
                        P.left->at[at] = make_int2(m + h, c);
                }
                continue;
            }
            double x;
            if (failed || sm == kNotFinite || sn == kNotFinite) {
                x = __longlong_as_double(0x7ff8000000000000ll);
            } else {
                x = limbs_double<N>(f, (int)(h ? q >> 32 : q) - 0x4b400000,
                                    P.alpha_exp - sm - sn);
                if (P.alpha_neg)
                    x = __longlong_as_double(__double_as_longlong(x) ^ (1ll << 63));
                if (P.alpha_mul)
                    x *= P.out.alpha;
            }
            if (P.beta_mode == 1)
                x += *dst;
            else if (P.beta_mode == 2)
                x += P.out.beta * *dst;
            *dst = x;
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static int get_encode(EncodeTiledFn *fn)
{
    static std::atomic<EncodeTiledFn> cached{nullptr};
    EncodeTiledFn f = cached.load();
    if (!f) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000,
                                                         cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !p) {
            cudaGetLastError();
            cutc_set_error(CUTC_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
            return CUTC_ERR_CUDA;
        }
        f = (EncodeTiledFn)p;
        cached.store(f);
    }
    *fn = f;
    return CUTC_OK;
}

int encode_bf16_map(CUtensorMap *map, const void *base, int rank, const uint64_t *dims,
                    const uint64_t *strides_bytes, const uint32_t *box, int swizzle)
{
    EncodeTiledFn enc;
    CUTC_TRY(get_encode(&enc));
    cuuint64_t d[3], s[2];
    cuuint32_t b[3] = {box[0], box[1], 1};
    cuuint32_t estr[3] = {1, 1, 1};
    for (int i = 0; i < rank; i++)
        d[i] = dims[i];
    for (int i = 0; i + 1 < rank; i++)
        s[i] = strides_bytes[i];
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void *>(base), d, s, b,
                     estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     swizzle == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        cutc_set_error(CUTC_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
        return CUTC_ERR_CUDA;
    }
    return CUTC_OK;
}

static int planes_map(CUtensorMap *map, int n_mod, const ResiduePlanes &o, int box_rows)
{
    const uint64_t dims[3] = {(uint64_t)o.kp, (uint64_t)o.rows, (uint64_t)n_mod};
    const uint64_t strides[2] = {(uint64_t)o.pitch * 2, (uint64_t)o.pitch * 2 * (uint64_t)o.rows};
    const uint32_t box[2] = {(uint32_t)kBK, (uint32_t)box_rows};
    return encode_bf16_map(map, o.p, 3, dims, strides, box, 128);
}

int modular_pass_cols(int n_mod, int64_t M, int64_t N, size_t out_bytes)
{
    const int64_t per = (int64_t)out_bytes / (2 * n_mod * modular_ldm(M));
    return (int)std::min<int64_t>(N, std::max<int64_t>(256, per / 256 * 256));
}

size_t modular_out_bytes(int n_mod, int64_t M, int64_t N, size_t out_bytes)
{
    return (size_t)2 * n_mod * modular_ldm(M) * modular_pass_cols(n_mod, M, N, out_bytes);
}

template <int BN, bool kResident, bool kMag>
static int launch_gemm(cudaStream_t st, const ResiduePlanes &A, const ResiduePlanes &B,
                       ModGemmParams P)
{
    using Cfg = ModCfg<BN>;
    static std::atomic<unsigned long long> attr_done{0};
    const unsigned long long bit = current_device_bit();
    if (!(attr_done.load() & bit)) {
        CUTC_CUDA_TRY(cudaFuncSetAttribute(modular_gemm_kernel<BN, kResident, kMag>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem));
        attr_done.fetch_or(bit);
    }
    CUtensorMap ta, tb;
    CUTC_TRY(planes_map(&ta, P.planes, A, 128));
    CUTC_TRY(planes_map(&tb, P.planes, B, BN / 2));
    P.tiles_m = (int)ceil_div(P.M, kTileM);
    P.tiles_n = (int)ceil_div(P.N, BN);
    const int64_t tasks = (int64_t)P.planes * P.tiles_m * P.tiles_n;
    if (tasks > INT32_MAX / 2) {
        cutc_set_error(CUTC_ERR_INVALID, "modular contraction of %lld tiles", (long long)tasks);
        return CUTC_ERR_INVALID;
    }
    const unsigned pairs = (unsigned)(kResident ? std::min<int64_t>(tasks, device_sms() / 2) : tasks);
    modular_gemm_kernel<BN, kResident, kMag><<<2 * pairs, kGemmThreads, Cfg::kSmem, st>>>(ta, tb, P);
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    return CUTC_OK;
}

int modular_gemm(cudaStream_t st, int n_mod, int planes, const ResiduePlanes &A, const ResiduePlanes &B,
                 unsigned short *out, int64_t plane_cols, bool accumulate, int *err)
{
    if (A.rows <= 0 || B.rows <= 0 || A.kp <= 0)
        return CUTC_OK;
    ModGemmParams P{};
    P.planes = planes;
    P.magnitudes = n_mod;
    P.M = A.rows;
    P.N = B.rows;
    P.nkb = (int)ceil_div(A.kp, kBK);
    P.accumulate = accumulate ? 1 : 0;
    P.out = out;
    P.ldm = modular_ldm(A.rows);
    P.plane = P.ldm * plane_cols;
    for (int i = 0; i < n_mod; i++) {
        P.p[i] = (float)moduli::prime(i);
        P.inv[i] = 1.0f / (float)moduli::prime(i);
    }
    P.err = err;
    // narrow tiles for few columns, and where wide ones would leave the SM pairs (76) short
    // of work
    const int64_t wide = (int64_t)planes * ceil_div(P.M, kTileM) * ceil_div(P.N, 256);
    const int bn = P.N <= 64 ? 64 : (P.N <= 128 || wide < device_sms() / 2) ? 128 : 256;
    // Short panels: resident pairs walk the tasks, which hides a task's set-up and epilogue
    // behind the next one's MMAs.  Long ones: one pair per task, which the hardware starts
    // in order, so that concurrent tasks stay neighbours in L2.  M 7260, N 16384, resident
    // against one by one: K 1024 1.71 / 2.85 ms, 4096 6.04 / 7.07, 16384 25.1 / 24.4.
    const bool resident = P.nkb <= kResidentBlocks, mag = planes > n_mod;
    auto launch = [&](auto width, auto res) {
        constexpr int BN = decltype(width)::value;
        constexpr bool kRes = decltype(res)::value;
        return mag ? launch_gemm<BN, kRes, true>(st, A, B, P) : launch_gemm<BN, kRes, false>(st, A, B, P);
    };
    auto widths = [&](auto res) {
        return bn == 64    ? launch(std::integral_constant<int, 64>{}, res)
               : bn == 128 ? launch(std::integral_constant<int, 128>{}, res)
                           : launch(std::integral_constant<int, 256>{}, res);
    };
    return resident ? widths(std::true_type{}) : widths(std::false_type{});
}

template <int N, bool kChecked = false>
static int launch_combine(cudaStream_t st, const CombineParams &P)
{
    dim3 grid(ceil_div(P.M, 256), (unsigned)std::min(P.ncols, 65535));
    combine_kernel<N, kChecked><<<grid, 128, 0, st>>>(P);
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    return CUTC_OK;
}

int modular_combine(cudaStream_t st, int n_mod, int M, int n0, int ncols, const unsigned short *res,
                    const int *sa, const int *sb, const ModularOut &out, const int *err,
                    LeftResults *left)
{
    if (M <= 0 || ncols <= 0)
        return CUTC_OK;
    CombineParams P;
    P.M = M;
    P.ncols = ncols;
    P.n0 = n0;
    P.res = res;
    P.ldm = modular_ldm(M);
    P.plane = P.ldm * ncols;
    P.sa = sa;
    P.sb = sb;
    P.out = out;
    // a power of two (1, -1/2, 1/2 in this library) scales through the exponent
    int ae = 0;
    const double am = std::frexp(std::fabs(out.alpha), &ae);
    P.alpha_mul = am != 0.5;
    P.alpha_exp = P.alpha_mul ? 0 : ae - 1;
    P.alpha_neg = !P.alpha_mul && out.alpha < 0;
    P.beta_mode = out.beta == 0.0 ? 0 : out.beta == 1.0 ? 1 : 2;
    P.err = err;
    P.left = left;
    if (left && n_mod == kPlainModuli)
        return launch_combine<kPlainModuli, true>(st, P);
    switch (left ? 0 : n_mod) {
    case 8: return launch_combine<8>(st, P);
    case 9: return launch_combine<9>(st, P);
    case 10: return launch_combine<10>(st, P);
    case 11: return launch_combine<11>(st, P);
    case 12: return launch_combine<12>(st, P);
    case 13: return launch_combine<13>(st, P);
    case 15: return launch_combine<15>(st, P);
    case 17: return launch_combine<17>(st, P);
    }
    cutc_set_error(CUTC_ERR_INVALID, "no combination of %d moduli", n_mod);
    return CUTC_ERR_INVALID;
}

}  // namespace cutc
