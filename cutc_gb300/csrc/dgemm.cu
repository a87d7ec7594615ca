// FP64 contractions: fp64_contract, the modular contraction at FP64's precision (below),
// and the FP64 GEMM of DMMA (mma.sync m8n8k4 .f64) tiles fed by a multi-stage cp.async
// pipeline, which takes contractions shorter than 16, operands with infinities or NaNs and
// cutc_fp64_gemm_dev.
//
// The contractions are the reference's cublasDgemm calls
// (src/build_int2_grad1_u12_ao.cu:152-159, src/build_int_2e_ao.cu:60-67 and 97-104):
//   X_m[p, r1] = sum_r2 P[p, r2] G_m[r1, r2]        (A K-contiguous, "OP_T")
//   H[p, q]    = sum_r1 X_3[p, r1] S0[q, r1]        (A M-contiguous, "OP_N")
//   N[p, l]    = -1/2 sum_{m, r1} X_m[p, r1] S_m[l, r1]
// GB300 executes FP64 at about 2 FMA per clock per SM (1.25 TFLOP/s for the
// chip), so the DMMA kernel is bound by the FP64 pipe and nothing else:
// a 128 x 128 x 16 tile step is 262 144 FMAs, ~130 000 clocks of one SM's
// FP64 pipe, against 32 KB of operands -- 0.25 B per clock of operand
// traffic, far below every memory limit.  What the kernel needs is the FP64
// pipe never idle: eight warps per CTA, each with 32 independent DMMAs per
// 4-wide K step (a 64 x 32 warp tile, 64 FP64 accumulators per thread), and
// the next operand tiles in flight (three cp.async stages) while the current
// one is consumed.  Operands are copied with 8-byte cp.async, whose only
// alignment rule is the element's own: the strides here (n_grid2, block
// rows, n_ao^2) are arbitrary, which rules out TMA's 16-byte stride rule, and
// the copy engine would buy nothing at this arithmetic intensity.
//
// Shared-memory tiles are padded so that the DMMA fragment loads (8 rows x 4 k
// per warp, 256 bytes) take the minimum two wavefronts: a K-contiguous
// operand is stored [row][k] with 20 doubles per row, an M-contiguous one
// [k][row] with 136 doubles per k.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "dgemm.cuh"
#include "modular.cuh"
#include "residue.cuh"

namespace cutc {

namespace {

constexpr int kBM = 128, kBN = 128, kBK = 16, kStages = 3, kThreads = 256;
constexpr int kLdRow = kBK + 4;               // [row][k] tiles
constexpr int kLdCol = kBM + 8;               // [k][row] tiles
constexpr int kTileRow = kBM * kLdRow;        // 2560 doubles
constexpr int kTileCol = kBK * kLdCol;        // 2176 doubles
constexpr int kStageA = kTileRow > kTileCol ? kTileRow : kTileCol;
constexpr int kStageB = kBN * kLdRow;
constexpr int kSmem = kStages * (kStageA + kStageB) * (int)sizeof(double);  // 120 KB
static_assert(kBM == kBN, "the loaders assume square CTA tiles");

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

// 8-byte asynchronous copy; src_bytes = 0 writes zeros (out-of-range elements)
__device__ __forceinline__ void cp_async8(uint32_t dst, const double *src, uint32_t src_bytes)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src),
                 "r"(src_bytes)
                 : "memory");
}

__device__ __forceinline__ void cp_async_commit()
{
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// d += a b over one 8 x 8 x 4 step: a = A[lane / 4][lane % 4] (row-major A),
// b = B[lane % 4][lane / 4] (column-major B), d = D[lane / 4][2 (lane % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

struct Args {
    int M, N;
    int64_t K;
    double alpha, beta;
    const double *A, *B;
    double *C;
    int64_t lda, ldb, ldc, sa, sb, sc;
    int tiles_m, tiles_n;
};

// acc[i][j][h]: element (wm 64 + 8 i + lane / 4, wn 32 + 8 j + 2 (lane % 4) + h) of the 128 x 128
// tile at (m0, n0) of A B, wm = warp % 2 and wn = warp / 2; smem: kSmem bytes.
template <bool AK>
__device__ __forceinline__ void tile_product(const double *A, int64_t lda, const double *B,
                                             int64_t ldb, int M, int N, int64_t K, int m0, int n0,
                                             double *smem, double (&acc)[8][4][2])
{
    double *sA = smem;                       // kStages x kStageA
    double *sB = smem + kStages * kStageA;   // kStages x kStageB
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t nkb = (K + kBK - 1) / kBK;

    auto load = [&](int stage, int64_t kb) {
        const int64_t k0 = kb * kBK;
        double *a = sA + stage * kStageA, *b = sB + stage * kStageB;
#pragma unroll
        for (int i = 0; i < kBM * kBK / kThreads; i++) {
            const int e = tid + kThreads * i;
            int row, k;
            if (AK) {
                row = e / kBK;
                k = e % kBK;
            } else {
                k = e / kBM;
                row = e % kBM;
            }
            const int gm = m0 + row;
            const int64_t gk = k0 + k;
            const bool ok = gm < M && gk < K;
            const double *src = ok ? (AK ? A + (int64_t)gm * lda + gk : A + gk * lda + gm) : A;
            cp_async8(smem_u32(AK ? a + row * kLdRow + k : a + k * kLdCol + row), src, ok ? 8u : 0u);
        }
#pragma unroll
        for (int i = 0; i < kBN * kBK / kThreads; i++) {
            const int e = tid + kThreads * i;
            const int row = e / kBK, k = e % kBK;
            const int gn = n0 + row;
            const int64_t gk = k0 + k;
            const bool ok = gn < N && gk < K;
            const double *src = ok ? B + (int64_t)gn * ldb + gk : B;
            cp_async8(smem_u32(b + row * kLdRow + k), src, ok ? 8u : 0u);
        }
    };

    // warp tile: rows wm * 64 .. + 64, columns wn * 32 .. + 32
    const int wm = warp & 1, wn = warp >> 1;
    const int fr = lane >> 2, fk = lane & 3;
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            acc[i][j][0] = acc[i][j][1] = 0.0;

#pragma unroll
    for (int s = 0; s < kStages - 1; s++) {
        if (s < nkb)
            load(s, s);
        cp_async_commit();
    }
    for (int64_t kb = 0; kb < nkb; kb++) {
        cp_async_wait<kStages - 2>();
        __syncthreads();  // stage kb landed for every thread; stage kb - 1 is free
        const int64_t pre = kb + kStages - 1;
        if (pre < nkb)
            load((int)(pre % kStages), pre);
        cp_async_commit();
        const int stage = (int)(kb % kStages);
        const double *a = sA + stage * kStageA, *b = sB + stage * kStageB;
#pragma unroll
        for (int kk = 0; kk < kBK / 4; kk++) {
            const int k = kk * 4 + fk;
            double av[8], bv[4];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int row = wm * 64 + i * 8 + fr;
                av[i] = AK ? a[row * kLdRow + k] : a[k * kLdCol + row];
            }
#pragma unroll
            for (int j = 0; j < 4; j++)
                bv[j] = b[(wn * 32 + j * 8 + fr) * kLdRow + k];
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++)
                    dmma(acc[i][j][0], acc[i][j][1], av[i], bv[j]);
        }
    }
    cp_async_wait<0>();
    __syncthreads();  // the stages are free
}

template <bool AK>
__global__ void __launch_bounds__(kThreads, 1) fp64_gemm_kernel(const Args g)
{
    extern __shared__ __align__(16) double smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t per_batch = (int64_t)g.tiles_m * g.tiles_n;
    const int64_t t = blockIdx.x;
    const int z = (int)(t / per_batch);
    const int64_t r = t - (int64_t)z * per_batch;
    const int m0 = (int)(r % g.tiles_m) * kBM;  // m fastest: a wave shares the B tiles
    const int n0 = (int)(r / g.tiles_m) * kBN;
    double *C = g.C + (int64_t)z * g.sc;
    double acc[8][4][2];
    tile_product<AK>(g.A + (int64_t)z * g.sa, g.lda, g.B + (int64_t)z * g.sb, g.ldb, g.M, g.N, g.K,
                     m0, n0, smem, acc);
    const int wm = warp & 1, wn = warp >> 1;
    const int fr = lane >> 2, fk = lane & 3;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int m = m0 + wm * 64 + i * 8 + fr;
        if (m >= g.M)
            continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int n = n0 + wn * 32 + j * 8 + 2 * fk + h;
                if (n < g.N) {
                    double *c = C + m + (int64_t)n * g.ldc;
                    const double v = g.alpha * acc[i][j][h];
                    *c = g.beta == 0.0 ? v : v + g.beta * *c;
                }
            }
        }
    }
}

// The results that a checked modular contraction left out (result_left), in FP64: M x N
// results of one pass, by a block per SM.  Listed ones are formed by a warp each (12 000 x 300
// results of K 12 000 with some dozens left: 0.70 ms when every block looked for its tiles'
// own, 0.04 so).  With more than the list holds, the blocks walk the 128 x 128 tiles and
// list each one's: up to kFewLeft are formed by a warp each, whose loads of 16 bytes per term
// the L2 feeds at about the FP64 pipe's rate, more by the whole tile's product.
struct RestArgs {
    int M, N;
    int64_t K;
    const double *A, *B;  // at the pass's first row and column
    int64_t lda, ldb;
    const unsigned short *sums;  // sums[n ldm + m]
    int64_t ldm;
    const int *sa, *sb;
    int n0;
    ModularOut out;
    const LeftResults *left;
};
constexpr int kFewLeft = 2048;

template <bool AK>
__global__ void __launch_bounds__(kThreads, 1) contract_rest_kernel(const RestArgs g)
{
    const int total = g.left->count;
    if (total == 0)
        return;
    extern __shared__ __align__(16) double smem[];
    __shared__ unsigned short s_list[kFewLeft];
    __shared__ int s_count;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tiles_m = (g.M + kBM - 1) / kBM, tiles_n = (g.N + kBN - 1) / kBN;
    auto left = [&](int m, int n) {
        return m < g.M && n < g.N &&
               result_left(g.sums[(int64_t)n * g.ldm + m], g.sa[m], g.sb[n]);
    };
    auto store = [&](int m, int n, double sum) {
        const ModularOut &o = g.out;
        const int gm = o.row0 + m, gn = g.n0 + n;
        const int64_t row = o.nrow_group ? (int64_t)(gm / o.nrow_group) * o.row_stride + gm % o.nrow_group
                                         : gm;
        const int64_t col = (int64_t)(gn / o.ncol_group) * o.group_stride + o.col0 + gn % o.ncol_group;
        double *c = o.C + row + o.ldc * col;
        const double v = o.alpha * sum;
        *c = o.beta == 0.0 ? v : v + o.beta * *c;
    };
    auto one = [&](int m, int n) {  // by a warp
        const double *a = AK ? g.A + (int64_t)m * g.lda : g.A + m;
        const double *b = g.B + (int64_t)n * g.ldb;
        double sum = 0.0;
#pragma unroll 8
        for (int64_t k = lane; k < g.K; k += 32)
            sum = fma(AK ? a[k] : a[k * g.lda], b[k], sum);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0)
            store(m, n, sum);
    };
    if (total <= kMaxListed) {
        // (the blocks take neighbours of the list in turn)
        for (int e = warp * gridDim.x + blockIdx.x; e < total; e += gridDim.x * (kThreads / 32)) {
            const int2 at = g.left->at[e];
            one(at.x, at.y);
        }
        return;
    }
    for (int64_t t = blockIdx.x; t < (int64_t)tiles_m * tiles_n; t += gridDim.x) {
        const int m0 = (int)(t % tiles_m) * kBM, n0 = (int)(t / tiles_m) * kBN;
        __syncthreads();  // the last tile's list is read
        if (threadIdx.x == 0)
            s_count = 0;
        __syncthreads();
        for (int k = threadIdx.x; k < kBM * kBN; k += kThreads)
            if (left(m0 + k % kBM, n0 + k / kBM)) {
                const int at = atomicAdd(&s_count, 1);
                if (at < kFewLeft)
                    s_list[at] = (unsigned short)k;
            }
        __syncthreads();
        const int count = s_count;
        if (count <= kFewLeft) {
            for (int e = warp; e < count; e += kThreads / 32)
                one(m0 + s_list[e] % kBM, n0 + s_list[e] / kBM);
            continue;
        }
        double acc[8][4][2];
        tile_product<AK>(g.A, g.lda, g.B, g.ldb, g.M, g.N, g.K, m0, n0, smem, acc);
        const int wm = warp & 1, wn = warp >> 1;
        const int fr = lane >> 2, fk = lane & 3;
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int m = m0 + wm * 64 + i * 8 + fr, n = n0 + wn * 32 + j * 8 + 2 * fk + h;
                    if (left(m, n))
                        store(m, n, acc[i][j][h]);
                }
    }
}

template <bool AK>
int launch_rest(cudaStream_t st, const RestArgs &g, int n_sm)
{
    static std::atomic<unsigned long long> attr_done{0};
    const unsigned long long bit = current_device_bit();
    if (!(attr_done.load() & bit)) {
        CUTC_CUDA_TRY(cudaFuncSetAttribute(contract_rest_kernel<AK>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        attr_done.fetch_or(bit);
    }
    const int64_t tiles = ((int64_t)g.M + kBM - 1) / kBM * (((int64_t)g.N + kBN - 1) / kBN);
    contract_rest_kernel<AK><<<(unsigned)std::min<int64_t>(tiles, n_sm), kThreads, kSmem, st>>>(g);
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    return CUTC_OK;
}

}  // namespace

int fp64_gemm(cudaStream_t st, bool a_kmajor, int M, int N, int64_t K, double alpha,
              const double *A, int64_t lda, int64_t sa, const double *B, int64_t ldb, int64_t sb,
              double beta, double *C, int64_t ldc, int64_t sc, int batch)
{
    if (M < 0 || N < 0 || K < 0 || batch < 0 || ldc < std::max(1, M) ||
        (K > 0 && (!A || !B || ldb < K || lda < (a_kmajor ? K : (int64_t)M))) || (M && N && !C)) {
        cutc_set_error(CUTC_ERR_INVALID, "invalid FP64 GEMM arguments (M=%d N=%d K=%lld)", M, N,
                       (long long)K);
        return CUTC_ERR_INVALID;
    }
    if (M == 0 || N == 0 || batch == 0)
        return CUTC_OK;
    static std::atomic<unsigned long long> attr_done{0};
    const unsigned long long bit = current_device_bit();
    if (!(attr_done.load() & bit)) {
        CUTC_CUDA_TRY(cudaFuncSetAttribute(fp64_gemm_kernel<true>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        CUTC_CUDA_TRY(cudaFuncSetAttribute(fp64_gemm_kernel<false>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        attr_done.fetch_or(bit);
    }
    Args g;
    g.M = M;
    g.N = N;
    g.K = K;
    g.alpha = alpha;
    g.beta = beta;
    g.A = A;
    g.B = B;
    g.C = C;
    g.lda = lda;
    g.ldb = ldb;
    g.ldc = ldc;
    g.sa = sa;
    g.sb = sb;
    g.sc = sc;
    g.tiles_m = (M + kBM - 1) / kBM;
    g.tiles_n = (N + kBN - 1) / kBN;
    const int64_t tiles = (int64_t)g.tiles_m * g.tiles_n * batch;
    if (tiles > INT32_MAX) {
        cutc_set_error(CUTC_ERR_INVALID, "FP64 GEMM of %lld tiles exceeds one grid",
                       (long long)tiles);
        return CUTC_ERR_INVALID;
    }
    if (a_kmajor)
        fp64_gemm_kernel<true><<<(unsigned)tiles, kThreads, kSmem, st>>>(g);
    else
        fp64_gemm_kernel<false><<<(unsigned)tiles, kThreads, kSmem, st>>>(g);
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    return CUTC_OK;
}

// ---------------------------------------------------------------------------
// FP64 contractions on the BF16 tensor cores
// ---------------------------------------------------------------------------
//
// GB300's FP64 pipe gives 1.1 TF/s; 17 residue products and one of magnitudes at about
// 1.8 PF/s of BF16 give about 100 TF/s.  The operands are rounded at 2^-70 of their row norms
// and nothing else until the result is rounded to FP64, where a sum of K FP64 terms rounds K
// times.  Where |a|_2 |b|_2 is so far above sum_k |a_k b_k| that this is not the smaller error
// (rows that hardly overlap), where an operand is not finite, the FP64 GEMM's kernel forms the
// result (modular.cuh, kCheckSum).  Below K = 16 the DMMA kernel does no more than one of its K steps
// (65 us a wave of tiles), which the modular contraction's launches do not beat.

constexpr int kMinContractK = 16;
constexpr size_t kMinContractBytes = (size_t)16 << 20;  // no smaller blocks are tried
enum ContractSlot { C_FLAGS, C_SCA, C_SCB, C_RA, C_RB, C_OUT };
static_assert(C_OUT + 1 == kContractSlots, "slots");

// How a contraction is cut to fit `limit` bytes: half for the residues of A's rows in a K
// panel, a quarter each for B's columns and for the results of a pass.  All of K if that
// fits, then K panels of whole 512-long chunks, then blocks of rows; never below 256 rows,
// 256 columns and one chunk.
struct ContractPlan {
    int64_t kp;
    ModularBlocks blk;
    size_t a_bytes, b_bytes, out_bytes;
};

static ContractPlan contract_plan(int64_t M, int64_t N, int64_t K, size_t limit)
{
    constexpr int n = kPlainPlanes;
    const size_t half = limit / 2, quarter = limit / 4;
    auto whole = [](size_t fit, int64_t all) {  // a multiple of 256, at least one, at most all
        return (int)std::min<int64_t>(all, std::max<int64_t>(256, (int64_t)(fit / 256 * 256)));
    };
    ContractPlan c;
    c.kp = K;
    if (residue_bytes(n, M, K) > half)
        c.kp = std::min<int64_t>(K, std::max<int64_t>(512, (int64_t)(half / residue_bytes(n, M, 16) * 16) /
                                                               512 * 512));
    c.blk.rows = residue_bytes(n, M, c.kp) > half ? whole(half / residue_bytes(n, 1, c.kp), M) : (int)M;
    const int64_t least = std::min<int64_t>(N, 256);  // columns of a pass
    if ((size_t)2 * n * modular_ldm(c.blk.rows) * least > quarter)
        c.blk.rows = whole(quarter / (2 * n * least), c.blk.rows);
    c.blk.pass = whole(quarter / (2 * n * modular_ldm(c.blk.rows)), N);
    c.blk.group = std::min(c.blk.pass, whole(quarter / residue_bytes(n, 1, c.kp), N));
    c.a_bytes = residue_bytes(n, c.blk.rows, c.kp);
    c.b_bytes = residue_bytes(n, c.blk.group, c.kp);
    c.out_bytes = (size_t)2 * n * modular_ldm(c.blk.rows) * c.blk.pass;
    return c;
}

size_t fp64_contract_bytes(int64_t M, int64_t N, int64_t K, size_t limit)
{
    const ContractPlan c = contract_plan(M, N, K, limit);
    return c.a_bytes + c.b_bytes + c.out_bytes + 4 * (size_t)(M + N);
}

int fp64_contract_begin(Workspace &W, int slot0, cudaStream_t st, size_t limit, ContractScratch &S)
{
    void *p;
    CUTC_TRY(W.get(slot0 + C_FLAGS, 64 + sizeof(LeftResults), &p));
    S.W = &W;
    S.limit = limit;
    S.slot0 = slot0;
    S.flags = (int *)p;
    S.left = (LeftResults *)((char *)p + 64);
    CUTC_CUDA_TRY(cudaMemsetAsync(p, 0, 64, st));
    return CUTC_OK;
}

int fp64_contract_check(const ContractScratch &S, cudaStream_t st)
{
    int err = 0;
    CUTC_CUDA_TRY(cudaMemcpyAsync(&err, S.flags, 4, cudaMemcpyDeviceToHost, st));
    CUTC_CUDA_TRY(cudaStreamSynchronize(st));
    if (err) {
        cutc_set_error(CUTC_ERR_TIMEOUT, "a tensor-core pipeline wait gave up (code %d)", err);
        return CUTC_ERR_TIMEOUT;
    }
    return CUTC_OK;
}

// A K-contiguous (rows lda apart) or M-contiguous (columns lda apart), B K-contiguous.
// *done is false, and nothing has run, when the device memory for the residues cannot be had
// even in the smallest blocks.
static int contract(const ContractScratch &S, cudaStream_t st, bool a_kmajor, int M, int N,
                    int64_t K, const double *A, int64_t lda, const double *B, int64_t ldb,
                    const ModularOut &out, bool *done)
{
    constexpr int n_mod = kPlainModuli;
    Workspace &W = *S.W;
    int *err = S.flags;
    LeftResults *left = S.left;
    ContractPlan c;
    ResiduePlanes a;
    void *b = nullptr, *res = nullptr, *psa = nullptr, *psb = nullptr;
    *done = false;
    for (size_t limit = S.limit;; limit /= 4) {
        c = contract_plan(M, N, K, limit);
        int s = W.get(S.slot0 + C_SCA, (size_t)M * 4, &psa);
        if (s == CUTC_OK)
            s = W.get(S.slot0 + C_SCB, (size_t)N * 4, &psb);
        if (s == CUTC_OK)
            s = W.get(S.slot0 + C_RA, c.a_bytes, &a.p);
        if (s == CUTC_OK)
            s = W.get(S.slot0 + C_RB, c.b_bytes, &b);
        if (s == CUTC_OK)
            s = W.get(S.slot0 + C_OUT, c.out_bytes, &res);
        if (s == CUTC_OK)
            break;
        if (s != CUTC_ERR_NO_MEMORY)
            return s;
        if (limit < kMinContractBytes)
            return CUTC_OK;
    }
    *done = true;
    int *sca = (int *)psa, *scb = (int *)psb;
    const int64_t pan = c.kp;
    const SrcDense sa{A, lda}, sb{B, ldb};
    if (a_kmajor)
        CUTC_TRY(row_scales(st, sa, M, K, pan, n_mod, sca));
    else
        CUTC_TRY(row_scales_cols(st, A, lda, M, K, n_mod, sca));
    CUTC_TRY(row_scales(st, sb, N, K, pan, n_mod, scb));
    return modular_contract_blocks(
        st, n_mod, M, N, K, pan, c.blk, a, b, false, (unsigned short *)res, sca, scb, out, err, left,
        [&](int m0, int rows, int64_t k0, int64_t kp, const ResiduePlanes &o) -> int {
            return a_kmajor ? residue_rows<n_mod, true>(st, sa, m0, rows, K, k0, kp, o.pitch, sca, o.p)
                            : residue_cols<n_mod, true>(st, A + m0, lda, rows, k0, kp, o.pitch,
                                                        sca + m0, o.p);
        },
        [&](int n0, int nc, int64_t k0, int64_t kp, const ResiduePlanes &o) {
            return residue_rows<n_mod, true>(st, sb, n0, nc, K, k0, kp, o.pitch, scb, o.p);
        },
        [&](int m0, int rows, int n0, int nc, const unsigned short *sums, const ModularOut &o) {
            RestArgs g;
            g.M = rows;
            g.N = nc;
            g.K = K;
            g.A = A + (a_kmajor ? (int64_t)m0 * lda : m0);
            g.B = B + (int64_t)n0 * ldb;
            g.lda = lda;
            g.ldb = ldb;
            g.sums = sums;
            g.ldm = modular_ldm(rows);
            g.sa = sca + m0;
            g.sb = scb + n0;
            g.n0 = n0;
            g.out = o;
            g.left = left;
            return a_kmajor ? launch_rest<true>(st, g, device_sms())
                            : launch_rest<false>(st, g, device_sms());
        });
}

int fp64_contract(const ContractScratch &S, cudaStream_t st, bool a_kmajor, int M, int N,
                  int64_t K, double alpha, const double *A, int64_t lda, int64_t sa,
                  const double *B, int64_t ldb, int64_t sb, double beta, double *C, int64_t ldc,
                  int64_t sc, int batch)
{
    const bool joined = batch == 1 || (sa == 0 && sb == (int64_t)N * ldb && sc % ldc == 0 &&
                                       (int64_t)N * batch <= INT32_MAX);
    if (K < kMinContractK || M <= 0 || N <= 0 || batch <= 0 || ldc < M || ldb < K ||
        lda < (a_kmajor ? K : (int64_t)M))  // (fp64_gemm refuses what it cannot take)
        return fp64_gemm(st, a_kmajor, M, N, K, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc,
                         batch);
    if (!joined) {
        for (int z = 0; z < batch; z++)
            CUTC_TRY(fp64_contract(S, st, a_kmajor, M, N, K, alpha, A + z * sa, lda, 0,
                                   B + z * sb, ldb, 0, beta, C + z * sc, ldc, 0, 1));
        return CUTC_OK;
    }
    bool done;
    CUTC_TRY(contract(S, st, a_kmajor, M, N * batch, K, A, lda, B, ldb,
                      ModularOut{C, ldc, N, batch > 1 ? sc / ldc : 0, 0, alpha, beta}, &done));
    return done ? CUTC_OK
                : fp64_gemm(st, a_kmajor, M, N, K, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc,
                            batch);
}

int fp64_contract_rows(const ContractScratch &S, cudaStream_t st, int M, int N, int64_t K,
                       const double *A, int64_t lda, const double *B, int64_t ldb, double *C,
                       int64_t ldc, int nrow_group, int64_t row_stride)
{
    bool done = false;
    if (K >= kMinContractK)
        CUTC_TRY(contract(S, st, true, M, N, K, A, lda, B, ldb,
                          ModularOut{C, ldc, N, 0, 0, 1.0, 0.0, nrow_group, row_stride}, &done));
    if (done)
        return CUTC_OK;
    // the groups of rows as a batch: C of group z starts z row_stride further
    return fp64_gemm(st, true, nrow_group, N, K, 1.0, A, lda, (int64_t)nrow_group * lda, B, ldb, 0,
                     0.0, C, ldc, row_stride, M / nrow_group);
}

}  // namespace cutc
