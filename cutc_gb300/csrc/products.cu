// Grid pair products, X expansion and int_2e assembly (sm_103a).
//
// The reference materialises the full nA^2 pair products
//   P[j + nA i][r2]  = w2 chi_i chi_j                       (src/long_range_integ.cu:39)
//   S0[j + nA i][r1] = w1 chi_i chi_j                       (src/short_range_integ_herm.cu:38)
//   S[j + nA i][m][r1] = w1 (chi_j d_m chi_i - chi_i d_m chi_j)   (src/short_range_integ_nonherm.cu:55)
// with one thread per grid point writing nA^2 values at stride n.  Here:
//   * P and S0 are symmetric in the AO pair, so only the lower triangle
//     (a >= b, tri_index) is built: half the memory and half the GEMM work;
//   * S is antisymmetric, so only the strict lower triangle is built;
//   * threads run along the grid index, so every store is coalesced.
// The symmetric/antisymmetric halves are recombined in assemble_int2e_kernel,
// which also performs the reference's A + A^T (src/add_trans_inplace.cu:2-21)
// without materialising A.
#include "common.cuh"
#include "products.cuh"

namespace cutc {

// out[tri(a, b) * ld + g] = w[g] chi_a(g) chi_b(g), b <= a, g in [0, n)
__global__ void sym_products_kernel(int n, int nA, const double *__restrict__ w,
                                    const double *__restrict__ chi, int64_t ld_chi,
                                    double *__restrict__ out, int64_t ld)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int a = blockIdx.y;
    if (g >= n)
        return;
    const double wa = w[g] * chi[(int64_t)a * ld_chi + g];
    for (int b = 0; b <= a; b++)
        out[tri_index(a, b, nA) * ld + g] = wa * chi[(int64_t)b * ld_chi + g];
}

// out[stri(c, d) * ld + m * n + g] = w (chi_c d_m chi_d - chi_d d_m chi_c), c > d
// aos is the (ld_aos, nA, 4) array seen from the first of the n grid points;
// component k of AO a at aos[(k * nA + a) * ld_aos + g].
__global__ void antisym_products_kernel(int n, int nA, const double *__restrict__ w,
                                        const double *__restrict__ aos, int64_t ld_aos,
                                        double *__restrict__ out, int64_t ld)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = blockIdx.y;
    if (g >= n)
        return;
    const int64_t comp = (int64_t)nA * ld_aos;
    const double wg = w[g];
    const double vc = aos[(int64_t)c * ld_aos + g];
    const double dc0 = aos[comp + (int64_t)c * ld_aos + g];
    const double dc1 = aos[2 * comp + (int64_t)c * ld_aos + g];
    const double dc2 = aos[3 * comp + (int64_t)c * ld_aos + g];
    for (int d = 0; d < c; d++) {
        const double vd = aos[(int64_t)d * ld_aos + g];
        double *o = out + stri_index(c, d, nA) * ld + g;
        o[0] = wg * (vc * aos[comp + (int64_t)d * ld_aos + g] - vd * dc0);
        o[n] = wg * (vc * aos[2 * comp + (int64_t)d * ld_aos + g] - vd * dc1);
        o[2 * (int64_t)n] = wg * (vc * aos[3 * comp + (int64_t)d * ld_aos + g] - vd * dc2);
    }
}

// X[m * xs + i * nA^2 + a + nA b] = Xp[m * ps + i * ldp + tri(max(a,b), min(a,b))] for rows
// i < n of the requested components m.
__global__ void expand_pairs_kernel(int n, int64_t rows, int nA, const double *__restrict__ Xp,
                                    int64_t ldp, int64_t ps, double *__restrict__ X, int64_t xs)
{
    const int64_t row = blockIdx.y + (int64_t)gridDim.y * blockIdx.z;
    if (row >= rows)
        return;
    // nA^2 < 2^30 (the build's argument checks): 32-bit index arithmetic, one division
    const int n2 = nA * nA;
    const int64_t m = row / n, i = row - m * n;
    const double *src = Xp + m * ps + i * ldp;
    double *dst = X + m * xs + i * n2;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n2; k += gridDim.x * blockDim.x) {
        const int b = k / nA, a = k - b * nA;
        dst[k] = src[a >= b ? tri_index(a, b, nA) : tri_index(b, a, nA)];
    }
}

// int_2e from the packed contractions
//   H[p + np q]  symmetric part  (p = tri(a,b), q = tri(c,d))
//   N[p + np l]  antisymmetric part, l = stri(max(c,d), min(c,d)), sign + if c > d:
// A[(a,b), (c,d)] = H[p, q] +- N[p, l], and the result A + A^T at rows (a,b) and columns
// (c,d).  With u+- = H[p, q] +- N[p, l(q)] and w+- = H[q, p] +- N[q, l(p)] for pairs a >= b
// and c >= d, the pair of pairs gives the four elements
//   (a,b),(c,d): u+ + w+    (a,b),(d,c): u- + w+    (b,a),(c,d): u+ + w-    (b,a),(d,c): u- + w-
// (one where the indices coincide).  One block takes 16 a x 16 b x 4 c and walks d: the two
// orientations of H and N are staged through shared memory, so that reads run along p or
// along q (32-byte runs and longer) and both (a,b) and (b,a) rows are written in 128-byte
// runs.  Bound by HBM and L2: H and N are read two to four times, 8 B written per element.
// 180 AOs: 20.5 ms with one 32 x 32 tile of A per block and a gather per element, 6.4 ms so
// (8 c per block: 6.9).
// Columns col = c + nA d with t0 <= d < t1 are written (out holds t0 first).  PSQT: element
// (p,q,s,t) goes where (p,s,q,t) would.
constexpr int kAsmA = 16, kAsmC = 4;
constexpr int kAsmRow = kAsmA + 1;                    // doubles per b of a tile
constexpr int kAsmPlane = kAsmA * kAsmRow + 2;        // ... per c (spreads c over the banks)
constexpr int kAsmTile = kAsmC * kAsmPlane;
constexpr size_t kAsmSmem = 4 * kAsmTile * sizeof(double);

template <bool PSQT>
__global__ void __launch_bounds__(kAsmA *kAsmA)
assemble_int2e_kernel(int nA, const double *__restrict__ H, const double *__restrict__ N, int t0,
                      int t1, int d_per, double *__restrict__ out)
{
    extern __shared__ double sm[];
    double *hp = sm, *np_ = sm + kAsmTile, *hq = sm + 2 * kAsmTile, *nq = sm + 3 * kAsmTile;
    // block x = (ia, ib), ib <= ia, packed as tri_index packs (rows ia of the triangle)
    int ia = (int)((sqrtf(8.0f * blockIdx.x + 1.0f) - 1.0f) * 0.5f);
    while ((ia + 1) * (ia + 2) / 2 <= (int)blockIdx.x)
        ia++;
    while (ia * (ia + 1) / 2 > (int)blockIdx.x)
        ia--;
    const int ib = (int)blockIdx.x - ia * (ia + 1) / 2;
    const int a0 = ia * kAsmA, b0 = ib * kAsmA, c0 = (int)blockIdx.y * kAsmC;
    const int c_end = min(nA, c0 + kAsmC);
    const int d0 = (int)blockIdx.z * d_per, d_end = min(d0 + d_per, c_end);  // d <= c
    const int64_t np = (int64_t)nA * (nA + 1) / 2, n = (int64_t)nA * nA;
    const int lo = threadIdx.x & 15, hi = threadIdx.x >> 4;
    const bool c_in = c_end > t0 && c0 < t1;  // some column (d, c) is wanted

    for (int d = d0; d < d_end; d++) {
        const bool d_in = d >= t0 && d < t1;
        if (!d_in && !c_in)
            continue;
        // all of a thread's loads are issued before the first is stored: along p, thread =
        // (a, b) and one c each; along q, thread = (c, one of 32 pairs) and 8 pairs
        double vh[kAsmC], vn[kAsmC], wh[kAsmC], wn[kAsmC];
        const int a = a0 + lo, b = b0 + hi, cq = c0 + (int)(threadIdx.x % kAsmC);
        const int64_t p = tri_index(a, b, nA), q = tri_index(cq, d, nA);
        const bool p_ok = a < nA && b <= a, q_ok = cq < c_end && cq >= d;
#pragma unroll
        for (int k = 0; k < kAsmC; k++) {
            const int c = c0 + k;
            const bool ok = p_ok && c < c_end && c >= d;
            vh[k] = ok ? H[p + np * tri_index(c, d, nA)] : 0.0;
            vn[k] = ok && c > d ? N[p + np * stri_index(c, d, nA)] : 0.0;
            const int pr = (int)(threadIdx.x / kAsmC) + kAsmA * kAsmA / kAsmC * k, pa = a0 + (pr & 15), pb = b0 + (pr >> 4);
            const bool okq = q_ok && pa < nA && pb <= pa;
            wh[k] = okq ? H[q + np * tri_index(pa, pb, nA)] : 0.0;
            wn[k] = okq && pa > pb ? N[q + np * stri_index(pa, pb, nA)] : 0.0;
        }
        __syncthreads();  // the previous d's tiles are read
#pragma unroll
        for (int k = 0; k < kAsmC; k++) {
            const int o = k * kAsmPlane + hi * kAsmRow + lo;
            hp[o] = vh[k];
            np_[o] = vn[k];
            const int pr = (int)(threadIdx.x / kAsmC) + kAsmA * kAsmA / kAsmC * k;
            const int oq = (int)(threadIdx.x % kAsmC) * kAsmPlane + (pr >> 4) * kAsmRow + (pr & 15);
            hq[oq] = wh[k];
            nq[oq] = wn[k];
        }
        __syncthreads();
        for (int c = max(c0, d); c < c_end; c++) {
            const bool both = c > d && c >= t0 && c < t1;  // column (d, c) too
            // element (x, y) of the row pair and column (s, t)
            auto put = [&](int x, int y, int s, int t, double v) {
                const int64_t o = PSQT ? x + (int64_t)nA * s + n * y + n * nA * (t - t0)
                                       : x + (int64_t)nA * y + n * (s + (int64_t)nA * (t - t0));
                out[o] = v;
            };
#pragma unroll
            for (int flip = 0; flip < 2; flip++) {
                // rows (a, b), consecutive threads along a; then (b, a), along b
                const int ta = flip ? hi : lo, tb = flip ? lo : hi;
                const int a = a0 + ta, b = b0 + tb;
                if (a >= nA || b > a || (flip && a == b))
                    continue;
                const int o = (c - c0) * kAsmPlane + tb * kAsmRow + ta;
                const double h = hp[o], m = np_[o];  // (N is zero for c == d, a == b)
                const double w = flip ? hq[o] - nq[o] : hq[o] + nq[o];
                const int x = flip ? b : a, y = flip ? a : b;
                if (d_in)
                    put(x, y, c, d, (h + m) + w);
                if (both)
                    put(x, y, d, c, (h - m) + w);
            }
        }
    }
}

int launch_sym_products(cudaStream_t st, int n, int nA, const double *w, const double *chi,
                        int64_t ld_chi, double *out, int64_t ld)
{
    if (n <= 0)
        return CUTC_OK;
    dim3 grid(ceil_div(n, 128), nA);
    sym_products_kernel<<<grid, 128, 0, st>>>(n, nA, w, chi, ld_chi, out, ld);
    CUTC_CUDA_TRY(cudaGetLastError());
    return CUTC_OK;
}

int launch_antisym_products(cudaStream_t st, int n, int nA, const double *w, const double *aos,
                            int64_t ld_aos, double *out, int64_t ld)
{
    if (n <= 0 || nA < 2)
        return CUTC_OK;
    dim3 grid(ceil_div(n, 128), nA);
    antisym_products_kernel<<<grid, 128, 0, st>>>(n, nA, w, aos, ld_aos, out, ld);
    CUTC_CUDA_TRY(cudaGetLastError());
    return CUTC_OK;
}

int launch_expand_pairs(cudaStream_t st, int n, int comps, int nA, const double *Xp, int64_t ldp,
                        int64_t ps, double *X, int64_t xs)
{
    const int64_t rows = (int64_t)n * comps;
    if (rows <= 0)
        return CUTC_OK;
    const int64_t nA2 = (int64_t)nA * nA;
    unsigned gx = ceil_div(nA2, 256);
    if (gx > 64)
        gx = 64;
    unsigned gy = rows < 65535 ? (unsigned)rows : 65535u;
    unsigned gz = ceil_div(rows, gy);
    expand_pairs_kernel<<<dim3(gx, gy, gz), 256, 0, st>>>(n, rows, nA, Xp, ldp, ps, X, xs);
    CUTC_CUDA_TRY(cudaGetLastError());
    return CUTC_OK;
}

int launch_assemble_int2e(cudaStream_t st, int nA, const double *H, const double *N, int c0,
                          int c1, bool psqt, double *out)
{
    const int n = nA * nA;
    if (c0 < 0 || c1 > n || c0 >= c1)
        return CUTC_OK;
    if (c0 % nA || c1 % nA) {
        cutc_set_error(CUTC_ERR_INVALID, "int_2e slab [%d, %d) is not a whole number of t", c0, c1);
        return CUTC_ERR_INVALID;
    }
    static std::atomic<unsigned long long> attr_done{0};
    const unsigned long long bit = current_device_bit();
    if (!(attr_done.load() & bit)) {
        CUTC_CUDA_TRY(cudaFuncSetAttribute(assemble_int2e_kernel<true>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, kAsmSmem));
        CUTC_CUDA_TRY(cudaFuncSetAttribute(assemble_int2e_kernel<false>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, kAsmSmem));
        attr_done.fetch_or(bit);
    }
    const int nb = (int)ceil_div(nA, kAsmA), nc = (int)ceil_div(nA, kAsmC);
    // d per block: fewer for small bases, which would not fill the SMs otherwise
    const int d_per = nA >= 64 ? 16 : 4;
    const dim3 grid((unsigned)(nb * (nb + 1) / 2), (unsigned)nc, ceil_div(nA, d_per));
    if (psqt)
        assemble_int2e_kernel<true><<<grid, kAsmA * kAsmA, kAsmSmem, st>>>(nA, H, N, c0 / nA, c1 / nA,
                                                                          d_per, out);
    else
        assemble_int2e_kernel<false><<<grid, kAsmA * kAsmA, kAsmSmem, st>>>(nA, H, N, c0 / nA, c1 / nA,
                                                                           d_per, out);
    CUTC_CUDA_TRY(cudaGetLastError());
    return CUTC_OK;
}

}  // namespace cutc
