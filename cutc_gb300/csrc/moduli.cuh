// Residue arithmetic of the modular contraction (modular.cu): the moduli, their tables
// and the scaling of operands to integers.
//
// An FP64 contraction C = A B^T is computed exactly on scaled, rounded operands,
//   t_a[m, k] = rint(A[m, k] 2^{s_m}),  t_b[n, k] = rint(B[n, k] 2^{u_n}),
// as the integers sum_k t_a t_b modulo N pairwise coprime odd moduli p_i <= 361.  A
// residue in [-180, 180] is an exact BF16 number and 512 products of two of them sum to
// less than 2^24 - 181, so the tensor cores' FP32 accumulation of a 512-long chunk is
// exact; the integer itself comes back from its N residues (Chinese remainder theorem) when
// |sum_k t_a t_b| < M / 2, M = prod p_i.  With row scales that bound the 2-norms,
// |t_a|_2, |t_b|_2 <= 2^beta(N), 2^{2 beta} < M / 2 (Cauchy-Schwarz), nothing else is
// rounded: the error is that of the operands' rounding, 2^-beta of their row norms,
// whatever K is.  One product per modulus replaces the S (S + 1) / 2 products of an
// S-slice splitting (Ozaki, Uchino and Imamura 2025, "Ozaki scheme II").  A slicing scales by
// the row's maximum, which a dense row's norm exceeds by up to sqrt(K): 12 or 13 products
// against the 15 of 5 slices have no coarser digits for any row (split_moduli), and
// 17 are needed for FP64's.  Larger moduli (<= 509, exact over 256 K) take
// one product fewer at FP64's error, but the accumulators' reads from tensor memory hold
// up the MMAs: M 7260, N 16384, K 16384 with 11 moduli took 33.5 ms in chunks of 256,
// 23.6 in chunks of 512.
#pragma once

#include <stdint.h>

#include "digits.cuh"

namespace cutc {
namespace moduli {

constexpr int kMax = 17;
constexpr int kChunkBits = 13;  // integers are cut into 13-bit chunks for the residues
constexpr int kMaxChunks = 6;

// Pairwise coprime, odd, <= 361: |residue| <= 180, running residues <= 181 (the FP32
// quotient S / p rounds to an integer one off only within 0.003 of a tie).
CUTC_HD constexpr int prime(int i)
{
    constexpr int p[kMax] = {361, 359, 355, 353, 351, 349, 347, 343,
                              341, 337, 331, 317, 313, 311, 307, 293, 289};
    return p[i];
}

// beta(n) = (log2(p_0 ... p_{n-1}) - 1) / 2, less 0.0125: the rows' log2 norm bound
CUTC_HD constexpr float row_bits(int n)
{
    constexpr float b[kMax + 1] = {0.f, 3.735f, 7.979f, 12.215f, 16.446f,
                                   20.674f, 24.898f, 29.117f, 33.328f, 37.535f,
                                   41.733f, 45.919f, 50.073f, 54.218f, 58.358f,
                                   62.489f, 66.587f, 70.674f};
    return b[n];
}

// 13-bit chunks that hold |t| <= 2^beta, below 2^{13 chunks - 1}
CUTC_HD constexpr int chunks(int n) { return n <= 9 ? 3 : n <= 11 ? 4 : n <= 15 ? 5 : 6; }

CUTC_HD constexpr int sym_mod(long long a, int p)  // in [-(p - 1) / 2, (p - 1) / 2]
{
    long long r = a % p;
    if (r < 0)
        r += p;
    return (int)(2 * r > p ? r - p : r);
}

CUTC_HD constexpr int inverse(int a, int p)  // a^-1 mod p (p small: by search)
{
    const int m = ((a % p) + p) % p;
    for (int x = 1; x < p; x++)
        if ((long long)m * x % p == 1)
            return sym_mod(x, p);
    return 0;
}

// |rint(x 2^s)| of an FP64 value (ties to even: rows of one sign gather no bias), in integer
// arithmetic, as T of 64 or 128 bits that hold it
template <class T>
CUTC_HD T scaled_magnitude(double x, int s)
{
    const unsigned long long bits = digits::double_bits(x);
    const int E = (int)((bits >> 52) & 0x7ff);
    const int sh = (E ? E : 1) - 1075 + s;
    const unsigned long long mant = (bits & ((1ull << 52) - 1)) | (E ? 1ull << 52 : 0ull);
    if (sh >= 0)
        return (T)mant << (sh & (8 * (int)sizeof(T) - 1));
    if (sh <= -54)
        return 0;
    return (T)((mant + ((1ull << (-sh - 1)) - 1) + ((mant >> -sh) & 1)) >> -sh);
}

}  // namespace moduli
}  // namespace cutc
