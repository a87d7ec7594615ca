// FP64 contractions of the plain form on the FP64 tensor path (DMMA).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "engine.cuh"

namespace cutc {

// C[m + ldc n] = alpha sum_k opA(m, k) B[n ldb + k] + beta C[m + ldc n]
// for m < M, n < N, over `batch` problems whose A, B and C start sa, sb and sc
// doubles apart.  opA(m, k) = A[m lda + k] when a_kmajor (K contiguous, cuBLAS
// OP_T on a K x M column-major array), else A[k lda + m] (M contiguous, OP_N).
// B is K contiguous per column n (OP_N on a K x N column-major array).  With
// beta == 0, C is not read.  Column-major C, as cuBLAS: the same call sites
// keep their argument meaning.
int fp64_gemm(cudaStream_t st, bool a_kmajor, int M, int N, int64_t K, double alpha,
              const double *A, int64_t lda, int64_t sa, const double *B, int64_t ldb, int64_t sb,
              double beta, double *C, int64_t ldc, int64_t sc, int batch);

// The same contraction for callers with a workspace: a checked modular contraction on the
// BF16 tensor cores (modular.cuh), whose operands' rounding adds less to any result than FP64
// sums round, with fp64_gemm's kernel for the results where it would not, for those of rows
// that hold an infinity or a NaN (both found on the device), and with fp64_gemm for K < 16.  S: from fp64_contract_begin; a
// bounded wait that gives up makes the results NaN and is reported by
// fp64_contract_check.  Batches whose A is common and whose B rows follow one another
// (sa = 0, sb = N ldb) are one contraction; others run one by one.
//
// Its residues take about `limit` bytes at most, whatever the sizes (contract_plan);
// where that memory cannot be had it takes less, and fp64_gemm's path without any in the end.
// The blocks do not change the results (but for which kernel gives those at the edge of the
// check).
//
// The scratch (kContractSlots slots from the given one) belongs to one stream until its
// work is done: calls that wait for their results share kContractSlot, a call that returns
// while its contractions still run has slots of its own.
struct LeftResults;
struct ContractScratch {
    Workspace *W = nullptr;
    int slot0 = 0;
    size_t limit = 0;
    int *flags = nullptr;  // [0]: a wait gave up
    LeftResults *left = nullptr;
};
constexpr size_t kContractBytes = (size_t)16 << 30;  // the largest limit
constexpr int kContractSlot = 100, kContractSlots = 6;
int fp64_contract_begin(Workspace &W, int slot0, cudaStream_t st, size_t limit, ContractScratch &S);
int fp64_contract(const ContractScratch &S, cudaStream_t st, bool a_kmajor, int M, int N,
                  int64_t K, double alpha, const double *A, int64_t lda, int64_t sa,
                  const double *B, int64_t ldb, int64_t sb, double beta, double *C, int64_t ldc,
                  int64_t sc, int batch);
// C[row(m) + ldc n] = sum_k A[m lda + k] B[n ldb + k] with rows in groups of nrow_group,
// row_stride apart (no batch).
int fp64_contract_rows(const ContractScratch &S, cudaStream_t st, int M, int N, int64_t K,
                       const double *A, int64_t lda, const double *B, int64_t ldb, double *C,
                       int64_t ldc, int nrow_group, int64_t row_stride);
int fp64_contract_check(const ContractScratch &S, cudaStream_t st);
// Device bytes fp64_contract keeps for operands of these sizes.
size_t fp64_contract_bytes(int64_t M, int64_t N, int64_t K, size_t limit);

}  // namespace cutc
