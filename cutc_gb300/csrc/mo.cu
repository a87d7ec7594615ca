// X in the molecular-orbital basis, in the order the reference's cutc_no reads it.
//
// cutc_int returns X in the AO basis as X_ao(a, b, g, m) (src/cutc_module.f90:34,
// column-major, AO pair fastest); cutc_no reads the MO-basis X as
// X_mo(g, m, i, j) with the grid point fastest (src/no_tmpJ_cs_kernel.cu:18-30,
// index g + n1 m + 3 n1 i + 3 n1 n_mo j).  The transform between them is done by
// the caller in the reference's workflow; here it is
//     X_mo(g, m, i, j) = sum_{a, b} L(a, i) X_ao(a, b, g, m) R(b, j)
// with L and R the left and right MO coefficients (n_ao x n_mo, column-major;
// L = R for a symmetric orbital set), in blocks of the points q = g + n1 m of all
// components, which are contiguous on both sides:
//     T(b, q, i)    = sum_a X(a, b, q) L(a, i)      rows (b, q), columns i
//     X_mo(q, i, j) = sum_b T(b, q, i) R(b, j)      rows (q, i), columns j
// Both are FP64 contractions of the plain form (dgemm.cuh) whose operands are K-contiguous
// and whose results are written in place, without a transpose: the short sides n_mo are
// the contractions' columns.  4 n_mo n_ao (n_ao + n_mo) n1 flops per component, bound by
// the operands' residues.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "dgemm.cuh"
#include "engine.cuh"

namespace cutc {

// (a device call returns while its work runs, so it shares no slot with other calls)
enum MoSlot { M_L = 180, M_R, M_T, M_XIN, M_XOUT, M_CONTRACT };

static int x_ao_to_mo(Engine *E, cudaStream_t st, int n1, int nA, int n_mo, int comps,
                      const double *L, const double *R, const double *x_ao, double *x_mo,
                      bool dev, size_t budget)
{
    Workspace &W = E->ws;
    void *p;
    const double *dL = L, *dR = R;
    const size_t cbytes = (size_t)nA * n_mo * 8;
    if (!dev) {
        CUTC_TRY(W.get(M_L, cbytes, &p));
        CUTC_CUDA_TRY(cudaMemcpyAsync(p, L, cbytes, cudaMemcpyHostToDevice, st));
        dL = (const double *)p;
        CUTC_TRY(W.get(M_R, cbytes, &p));
        CUTC_CUDA_TRY(cudaMemcpyAsync(p, R, cbytes, cudaMemcpyHostToDevice, st));
        dR = (const double *)p;
    }
    // points per block: T (and the host-mode staging of X_ao and X_mo); the contraction's
    // rows (b, q) and (q, i) are counted in 31 bits
    const size_t per_g = ((size_t)n_mo * nA + (dev ? 0 : (size_t)nA * nA + (size_t)n_mo * n_mo)) * 8;
    const int64_t nq = (int64_t)comps * n1;
    const int64_t cap = std::max<int64_t>(1, ((int64_t)1 << 28) / std::max(nA, n_mo));
    const int nb = (int)std::max<int64_t>(
        1, std::min<int64_t>(std::min(nq, cap), (int64_t)(budget / per_g)));
    double *T, *Xin = nullptr, *Xout = nullptr;
    CUTC_TRY(W.get(M_T, (size_t)n_mo * nA * nb * 8, &p));
    T = (double *)p;
    if (!dev) {
        CUTC_TRY(W.get(M_XIN, (size_t)nA * nA * nb * 8, &p));
        Xin = (double *)p;
        CUTC_TRY(W.get(M_XOUT, (size_t)n_mo * n_mo * nb * 8, &p));
        Xout = (double *)p;
    }
    ContractScratch contract;
    CUTC_TRY(fp64_contract_begin(W, M_CONTRACT, st, 4 * budget, contract));
    const int64_t nA2 = (int64_t)nA * nA, nm2 = (int64_t)n_mo * n_mo;
    for (int64_t q0 = 0; q0 < nq; q0 += nb) {
        const int qb = (int)std::min<int64_t>(nb, nq - q0);
        const double *X = x_ao + q0 * nA2;  // (a, b, q) of this block
        if (!dev) {
            CUTC_CUDA_TRY(cudaMemcpyAsync(Xin, X, (size_t)qb * nA2 * 8, cudaMemcpyHostToDevice, st));
            X = Xin;
        }
        // T[(b + nA q) + nA qb i]
        CUTC_TRY(fp64_contract(contract, st, true, nA * qb, n_mo, nA, 1.0, X, nA, 0, dL, nA, 0, 0.0,
                               T, (int64_t)nA * qb, 0, 1));
        // X_mo[q + ld (i + n_mo j)], rows m = q + qb i
        double *out = dev ? x_mo + q0 : Xout;
        const int64_t ld = dev ? nq : qb;
        CUTC_TRY(fp64_contract_rows(contract, st, n_mo * qb, n_mo, nA, T, nA, dR, nA, out,
                                    ld * n_mo, qb, ld));
        if (!dev)
            CUTC_CUDA_TRY(cudaMemcpy2DAsync(x_mo + q0, (size_t)nq * 8, Xout, (size_t)qb * 8,
                                            (size_t)qb * 8, (size_t)nm2, cudaMemcpyDeviceToHost, st));
    }
    // (device calls stay asynchronous: a wait that gave up shows as NaN results)
    if (!dev)
        CUTC_TRY(fp64_contract_check(contract, st));
    return CUTC_OK;
}

}  // namespace cutc

extern "C" int cutc_x_ao_to_mo(int n_grid1, int n_ao, int n_mo, int components,
                               const double *mo_l_coef, const double *mo_r_coef,
                               const double *x_ao, double *x_mo, int device_pointers, void *stream)
{
    using namespace cutc;
    if (n_grid1 <= 0 || n_ao <= 0 || n_mo <= 0 || (components != 3 && components != 4) ||
        !mo_l_coef || !mo_r_coef || !x_ao || !x_mo) {
        cutc_set_error(CUTC_ERR_INVALID, "invalid AO-to-MO arguments");
        return CUTC_ERR_INVALID;
    }
    if ((int64_t)n_mo * n_mo > INT32_MAX / 2 || (int64_t)n_ao * n_ao > INT32_MAX / 2) {
        cutc_set_error(CUTC_ERR_INVALID, "n_ao or n_mo too large");
        return CUTC_ERR_INVALID;
    }
    Engine *E = nullptr;
    CUTC_TRY(get_engine(&E));
    std::lock_guard<std::mutex> lk(E->mu);
    cudaStream_t st = stream ? (cudaStream_t)stream : E->stream;
    // the scratch may still be in use by a transform on another stream (a captured call's
    // order is that of its graph)
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CUTC_CUDA_TRY(cudaStreamIsCapturing(st, &cap));
    const bool eager = cap == cudaStreamCaptureStatusNone;
    if (eager && E->mo_used)
        CUTC_CUDA_TRY(cudaStreamWaitEvent(st, E->mo_done, 0));
    int s = x_ao_to_mo(E, st, n_grid1, n_ao, n_mo, components, mo_l_coef, mo_r_coef, x_ao, x_mo,
                       device_pointers != 0, (size_t)2 << 30);
    if (s == CUTC_OK && eager) {
        CUTC_CUDA_TRY(cudaEventRecord(E->mo_done, st));
        E->mo_used = true;
    }
    if (s != CUTC_OK)
        cudaStreamSynchronize(st);
    return s;
}
