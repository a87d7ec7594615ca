// Pair terms on the tensor cores: plan and entry points (pair_tc.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "engine.cuh"
#include "pair.cuh"

namespace cutc {

// One FP64 operand of the pair contraction as S BF16 slices [S][Mpad][Kpad] plus row
// exponents.
struct SliceOperand {
    void *sl = nullptr;  // __nv_bfloat16 slices
    int *ex = nullptr;   // row exponents (Mpad)
    int M = 0, Mpad = 0;
    int64_t K = 0, Kpad = 0;
};

// How a build's pair terms run on the tensor cores.
struct PairTcMode {
    int rows = 0;      // coefficient rows per r1 point: 16 (exponents in {0, 2, 3, 4}) or 32
                       // (any in [0, 6]); 0: not on the tensor cores
    int slices = 5;    // BF16 slices per operand: 5 or 6 (double-float results), 7 (FP64)
    bool fp64 = false; // FP64 results
    bool checked = false;  // results whose error may be above a term by term sum's are marked
    int powers() const { return rows == 16 ? 4 : 7; }
};

// The mode for a term table: double-float results from `slices` slices, or
// FP64 results.  rows == 0 where the tensor-core kernel does not apply (a coefficient that
// is not finite, or a kernel chosen by CUTC_PAIR_DF / CUTC_PAIR_DENSE for the double-float
// form).
PairTcMode pair_tc_mode(const double *coef, const int *exps, int n_terms, int n_nuc, bool fp64,
                        int slices);

struct PairTcPlan {
    PairTcMode mode;
    SliceOperand AF, BC;        // powers of f2 on r2; a tile's coefficient rows
    double *Fd = nullptr, *Cd = nullptr;
    float2 *r1d = nullptr;      // the tile's r1 points in double-float
    float *bscale = nullptr;    // 2^(row exponent) of the coefficient rows
    void *part = nullptr;       // the V values between the groups of a long contraction
    int64_t tile_rows = 0;      // r1 rows taken at once
    int *marked = nullptr;      // checked: set when pairs are left out; their bits 16 ints on
    int *err = nullptr;         // device flag set by a bounded wait that gave up
};

// Builds the F operand (powers of f2 on the n2 r2 points; f2 is [n_nuc][n2] FP64) and
// reserves the coefficient operand for tiles of up to n1t rows, taken in sub-tiles whose
// operands stay within kPairScratch and `scratch` bytes.  err: the caller's flag.
constexpr size_t kPairScratch = (size_t)2 << 30;
int pair_tc_prepare(Workspace &W, int slot0, cudaStream_t st, const PairTcMode &mode, int n2,
                    int n_nuc, const double *f2, int64_t n1t, size_t scratch, int *err,
                    PairTcPlan &plan);
// r2 points whose F operand takes about kPairScratch bytes.
int pair_tc_window(const PairTcMode &mode, int n_nuc);
// The pair planes of one r1 tile.  Double-float: P.G as for launch_pair_df.
int pair_tc_tile_df(cudaStream_t st, PairTcPlan &plan, const PairDfArgs &P, const double *rn,
                    double a_en, int n_sm);
// FP64: P.G as for launch_pair_f64 (P.t1 is not used), pairs that the check leaves out term by
// term.
int pair_tc_tile_f64(cudaStream_t st, PairTcPlan &plan, const PairArgs &P, const double *rn,
                     double a_en, int n_sm);
// Device bytes: fixed (F) and per r1 row of a tile, for the largest operands of the form.
size_t pair_tc_fixed_bytes(int n2, int n_nuc, int slices, size_t scratch);
size_t pair_tc_row_bytes(int n_nuc, int slices);

}  // namespace cutc
