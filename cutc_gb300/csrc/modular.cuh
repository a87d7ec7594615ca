// Modular contraction on the tensor cores: residue operands and entry points
// (moduli.cuh has the arithmetic, residue.cuh the operand preparation).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "engine.cuh"
#include "moduli.cuh"

namespace cutc {

// Row scale of a row that holds an infinity or a NaN.
constexpr int kNotFinite = INT32_MIN;

// Device tables of the moduli: FP32 pairs (both lanes the same value) for f32x2.
struct ModuliTab {
    uint64_t chunk[moduli::kMax][moduli::kMaxChunks];  // 2^{13 j} mod p_i
    uint64_t inv[moduli::kMax];                        // 1 / p_i
    uint64_t negp[moduli::kMax];                       // -p_i
};

constexpr uint32_t float_code(int v)  // the bits of a small integer as a float
{
    if (v == 0)
        return 0;
    const uint32_t sign = v < 0 ? 0x80000000u : 0u;
    uint32_t a = (uint32_t)(v < 0 ? -v : v);
    int e = 0;
    for (uint32_t t = a; t > 1; t >>= 1)
        e++;
    return sign | ((uint32_t)(127 + e) << 23) | ((a << (23 - e)) & 0x7fffffu);
}

constexpr uint32_t inverse_code(int p)  // 1 / p rounded to nearest, 256 < p < 512
{
    // 1 / p = f 2^-9 with 1 < f < 2: 24-bit significand round(2^32 / p)
    const uint64_t f = ((1ull << 32) + p / 2) / p;
    return (uint32_t)((127 - 9) << 23) | ((uint32_t)f & 0x7fffffu);
}

constexpr uint64_t dup_code(uint32_t c) { return ((uint64_t)c << 32) | c; }

constexpr ModuliTab make_moduli_tab()
{
    ModuliTab t{};
    for (int i = 0; i < moduli::kMax; i++) {
        const int p = moduli::prime(i);
        long long w = 1;
        for (int j = 0; j < moduli::kMaxChunks; j++) {
            t.chunk[i][j] = dup_code(float_code(moduli::sym_mod(w, p)));
            w = w * (1 << moduli::kChunkBits) % p;
        }
        t.inv[i] = dup_code(inverse_code(p));
        t.negp[i] = dup_code(float_code(-p));
    }
    return t;
}

static __constant__ const ModuliTab c_tab = make_moduli_tab();

// Moduli of a contraction over K columns with the precision of S 9-bit slices (3 .. 7).  S
// slices round a row at 2^-9S of a power of two above its maximum; here it is rounded at
// 2^-beta of its norm (to within a factor of 2, on both sides), at most sqrt(K) maxima.  With
// beta >= 9 S + log2(K) / 2 no row of any kind has a coarser unit than its slices had.  Of the
// numbers of moduli that are built; 7 slices beyond K = 41 000 keep 17, whose error stays
// below that of the products which slices leave out (s + t >= S) up to K = 1.6e5, and below
// FP64's rounding of the sum.
inline int split_moduli(int S, int64_t K)
{
    const float need = 9.0f * (float)S + 0.5f * log2f((float)std::max<int64_t>(K, 1));
    for (int n : {8, 9, 10, 11, 12, 13, 15})
        if (moduli::row_bits(n) >= need)
            return n;
    return moduli::kMax;
}
// Moduli of the plain form's contractions: operands rounded at 2^-70 of their row norms.  That
// is an error relative to |a|_2 |b|_2, where an FP64 sum's is relative to sum_k |a_k b_k|, so
// a checked contraction forms that sum too, in one more product of the operands' magnitudes
// (plane kPlainModuli, 8 bits of each), and leaves the results for which its error is not the
// smaller one to the FP64 GEMM.
//
// With t the operands' integers, |t|_2 <= 2^70.674, the rounding of both makes an error of at
// most 2^70.674 / sqrt(6) (rms, in units of the integer result).  Magnitudes enter as
// |t| 2^-58, so that the plane's sum is s = sum |t_a t_b| 2^-116, and with s >= kCheckSum
// that error is at most 0.17 2^-53 sum_k |a_k b_k|, about half of one rounding of an FP64
// sum (0.34 where the sum is of many K panels, each of which rounds it).  Sums are kept up to
// kMagnitudeCap; exact zeros (no k with both operands non-zero)
// are told from small ones, because their results are exact.  With 15 moduli, 2^-62, the
// check would fail for up to 8 % of the elements of a build (10 nuclei, 70 AOs: P against G's
// -1/2 |grad u|^2); with 17 for fewer than one in 10^5.
constexpr int kPlainModuli = moduli::kMax;
constexpr int kPlainPlanes = kPlainModuli + 1;
constexpr int kMagnitudeShift = 58, kMagnitudeCap = 32000, kCheckSum = 512;

// BF16 residues of one K panel of an operand: planes[i][r][k], rows `pitch` apart.
struct ResiduePlanes {
    void *p = nullptr;
    int rows = 0;
    int64_t kp = 0, pitch = 0;
};

// Where a contraction goes: C[row(m) + ldc col(n)] = alpha sum_k A[m, k] B[n, k] + beta C,
// col(n) = (n / ncol_group) group_stride + col0 + n % ncol_group, and with M = row0 + m
// row(m) = (M / nrow_group) row_stride + M % nrow_group (nrow_group 0: row(m) = M).
struct ModularOut {
    double *C;
    int64_t ldc;
    int ncol_group;
    int64_t group_stride, col0;
    double alpha, beta;
    int nrow_group = 0;
    int64_t row_stride = 0;
    int row0 = 0;
};

// Elements between the rows of a K panel of kp columns (whole 32-byte sectors; TMA takes
// multiples of 16 bytes).
inline int64_t residue_pitch(int64_t kp) { return (kp + 15) / 16 * 16; }

// Bytes of the residues of a panel (n_mod: its planes).
inline size_t residue_bytes(int n_mod, int64_t rows, int64_t kp)
{
    return (size_t)n_mod * rows * residue_pitch(kp) * 2;
}

// Columns per pass of a contraction with M rows: the residues of the results of one pass
// (2 bytes each and modulus) take at most out_bytes (one tile's columns at least).
int modular_pass_cols(int n_mod, int64_t M, int64_t N, size_t out_bytes);
size_t modular_out_bytes(int n_mod, int64_t M, int64_t N, size_t out_bytes);

// One K panel: residues of sum_k A[m, k] B[n, k] over the panel, for m < A.rows and
// n < B.rows, into out[i][n][m] (rows modular_ldm(A.rows) apart, planes plane_cols rows),
// added to what is there when accumulate.  err: set when a bounded wait gave up.  planes:
// n_mod, or n_mod + 1 with the magnitudes' sums (plane n_mod).
inline int64_t modular_ldm(int64_t M) { return (M + 7) / 8 * 8; }
int modular_gemm(cudaStream_t st, int n_mod, int planes, const ResiduePlanes &A, const ResiduePlanes &B,
                 unsigned short *out, int64_t plane_cols, bool accumulate, int *err);

// Results that a checked contraction leaves out of one pass.
constexpr int kMaxListed = 1 << 15;
struct LeftResults {
    int count;             // may exceed kMaxListed
    int2 at[kMaxListed];   // (row, column) in the pass's block
};

// The FP64 results from the residues: n0 .. n0 + ncols of the output's columns; sa and sb
// are the row scales of A and B (sb of column n0 first).  A result with a scale of
// kNotFinite, or after a wait that gave up, is NaN.  Checked (left not null, res with the
// magnitudes' sums): results of such scales and those whose sum is below kCheckSum are not
// written but counted and listed (result_left tells which, where the list is too short).
int modular_combine(cudaStream_t st, int n_mod, int M, int n0, int ncols, const unsigned short *res,
                    const int *sa, const int *sb, const ModularOut &out, const int *err,
                    LeftResults *left);

// A plane's entry for a magnitudes' sum, and whether a checked result is left out.
constexpr unsigned kResidueOffset = 512;
__device__ __forceinline__ bool result_left(unsigned entry, int sm, int sn)
{
    const unsigned c = entry - kResidueOffset;
    return sm == kNotFinite || sn == kNotFinite || (c != 0 && c < (unsigned)kCheckSum);
}

// cuTensorMapEncodeTiled of BF16 arrays: box[0] x box[1] tiles of the last two
// dimensions; swizzle in bytes (64 or 128).
int encode_bf16_map(CUtensorMap *map, const void *base, int rank, const uint64_t *dims,
                    const uint64_t *strides_bytes, const uint32_t *box, int swizzle);

// Rows of B whose residues of a K panel fit b_bytes (at least one tile's).
inline int modular_b_rows(int n_mod, int64_t N, int64_t kp, size_t b_bytes)
{
    const int64_t fit = (int64_t)(b_bytes / residue_bytes(n_mod, 1, kp)) / 256 * 256;
    return (int)std::min<int64_t>(N, std::max<int64_t>(256, fit));
}

// True when B's residues are whole in the workspace after the contraction.
inline bool modular_whole(int n_mod, int64_t N, int64_t K, int64_t k_panel, size_t b_bytes)
{
    return K <= k_panel && modular_b_rows(n_mod, N, K, b_bytes) >= N;
}

// How a contraction is cut: rows of A whose residues are in memory at once, columns of B
// likewise, and columns of results per pass.
struct ModularBlocks {
    int rows, group, pass;
};

// The contraction over K panels, gen_a(m0, rows, k0, kp, planes) and
// gen_b(n0, ncols, k0, kp, planes) writing the residues of a panel; gen_a may point planes.p
// at residues that are there already.  a.p, b_p and res: space for the residues of
// blk.rows x k_panel, blk.group x k_panel and of the results of one pass.  b_ready: B's are
// in b_p already (whole: k_panel >= K, blk.group >= N).  With left the contraction is checked:
// rest(m0, rows, n0, ncols, sums, out) is called after each pass for the results left out
// (sums: the magnitudes' plane, [n][m]).
template <class GenA, class GenB, class Rest>
int modular_contract_blocks(cudaStream_t st, int n_mod, int M, int N, int64_t K, int64_t k_panel,
                            const ModularBlocks &blk, ResiduePlanes a, void *b_p, bool b_ready,
                            unsigned short *res, const int *sa, const int *sb, ModularOut out,
                            int *err, LeftResults *left, GenA gen_a, GenB gen_b, Rest rest)
{
    const int planes = n_mod + (left ? 1 : 0);
    ResiduePlanes b;
    b.p = b_p;
    const bool b_whole = k_panel >= K && blk.group >= N && blk.pass >= N;
    for (int m0 = 0; m0 < M; m0 += blk.rows) {
        a.rows = std::min(blk.rows, M - m0);
        out.row0 = m0;
        bool a_ready = false;  // A's only panel stays for every pass
        for (int n0 = 0; n0 < N; n0 += blk.pass) {
            const int nc = std::min(blk.pass, N - n0);
            for (int64_t k0 = 0; k0 < K; k0 += k_panel) {
                const int64_t kp = std::min(k_panel, K - k0);
                a.kp = b.kp = kp;
                a.pitch = b.pitch = residue_pitch(kp);
                if (!a_ready)
                    CUTC_TRY(gen_a(m0, a.rows, k0, kp, a));
                a_ready = a_ready || k_panel >= K;
                for (int g = 0; g < nc; g += blk.group) {
                    b.rows = std::min(blk.group, nc - g);
                    if (!b_ready)
                        CUTC_TRY(gen_b(n0 + g, b.rows, k0, kp, b));
                    b_ready = b_ready || b_whole;
                    CUTC_TRY(modular_gemm(st, n_mod, planes, a, b, res + (int64_t)g * modular_ldm(a.rows),
                                          nc, k0 > 0, err));
                }
            }
            if (left)
                CUTC_CUDA_TRY(cudaMemsetAsync(&left->count, 0, sizeof(int), st));
            CUTC_TRY(modular_combine(st, n_mod, a.rows, n0, nc, res, sa + m0, sb + n0, out, err,
                                     left));
            if (left)
                CUTC_TRY(rest(m0, a.rows, n0, nc, res + (int64_t)n_mod * nc * modular_ldm(a.rows),
                              out));
        }
    }
    return CUTC_OK;
}

// The same with all rows of A at once and B's in groups of columns whose residues fit
// b_bytes and those of a pass of results out_bytes, the buffers from the workspace.
template <class GenA, class GenB>
int modular_contract(cudaStream_t st, Workspace &W, int slot_b, int slot_out, size_t b_bytes,
                     size_t out_bytes, int n_mod, int M, int N, int64_t K, int64_t k_panel, ResiduePlanes a,
                     bool b_ready, const int *sa, const int *sb,
                     const ModularOut &out, int *err, GenA gen_a, GenB gen_b)
{
    if (M <= 0 || N <= 0)
        return CUTC_OK;
    ModularBlocks blk;
    blk.rows = M;
    blk.pass = modular_pass_cols(n_mod, M, N, out_bytes);
    blk.group = std::min(blk.pass, modular_b_rows(n_mod, N, std::min(K, k_panel), b_bytes));
    void *b, *res;
    CUTC_TRY(W.get(slot_b, residue_bytes(n_mod, b_ready ? N : blk.group, std::min(K, k_panel)), &b));
    CUTC_TRY(W.get(slot_out, modular_out_bytes(n_mod, M, N, out_bytes), &res));
    return modular_contract_blocks(st, n_mod, M, N, K, k_panel, blk, a, b, b_ready,
                                   (unsigned short *)res, sa, sb, out, err, nullptr, gen_a, gen_b,
                                   [](int, int, int, int, const unsigned short *, const ModularOut &) {
                                       return CUTC_OK;
                                   });
}

}  // namespace cutc
