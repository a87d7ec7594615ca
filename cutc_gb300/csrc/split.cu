// The split form's contractions (modular.cu) and their operands.
//
// Both dense contractions of the cutc_int path
//   X_m[p, r1] = sum_r2 P[p, r2] G_m[r1, r2]                    (X build)
//   H[p, q] = sum_r1 X_3[p, r1] S0[q, r1],
//   N[p, l] = -1/2 sum_{m, r1} X_m[p, r1] S_m[l, r1]          (int_2e)
// are C[M x N] = alpha * A[M x K] B[N x K]^T with FP64 operands and run as modular
// contractions: exact integer products of the operands rounded on their row scales,
// one BF16 tensor-core product per modulus (moduli.cuh).  n_slices and K choose the number
// of moduli (split_moduli): the precision of at least that many 9-bit slices.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "products.cuh"
#include "residue.cuh"
#include "split.cuh"
#include "tc.cuh"

namespace cutc {

constexpr int kBK = 32;         // launches take whole blocks of 32 K
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

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

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
    SS_WCHI2, SS_WCHI1,
};

// K panel of a contraction (one launch's K).
static int64_t panel_k(int64_t K, int64_t M, int k_split)
{
    return std::min(K, (int64_t)split_k_blocks_per_launch(K, M, k_split) * kBK);
}

// The bytes below follow the build's scratch limit (R.scratch, half of its tile budget).
//
// Device bytes for the residues of B's columns: as many as the G tile they are formed
// from takes (its rows are then read once per panel, in a few groups of columns), at
// least 1 GiB if the limit allows, so that small contractions run in one group.
static size_t min_residue_bytes(const Request &R) { return std::min((size_t)1 << 30, R.scratch); }
static size_t x_residue_bytes(const Request &R, int64_t rows)
{
    return std::max(min_residue_bytes(R), (size_t)rows * 4 * (size_t)R.n2 * 8);
}
// Device bytes of each operand's residues in the int_2e contractions, and of a pass of results.
static size_t operand_bytes(const Request &R) { return std::min((size_t)4 << 30, R.scratch / 2); }

// K panel of the int_2e contractions: whole tensor-core chunks (256) whose residues of the
// np rows of A fit.
static int64_t int2e_panel_k(const Request &R, int n_mod, int64_t K, int64_t np)
{
    const int64_t fit = (int64_t)(operand_bytes(R) / (2 * (size_t)n_mod * np)) / 256 * 256;
    const int64_t cap = R.k_split > 0 ? panel_k(K, np, R.k_split) : K;
    return std::min(cap, std::max<int64_t>(256, fit));
}

// P's residues stay for every r1 tile (and, in a scan, for every set) when all K panels
// take at most 16 GiB and twice the limit; otherwise each tile forms a panel again (medium
// build, 7260 x 80 000: 3 ms a tile).
static size_t resident_bytes(const Request &R) { return std::min((size_t)16 << 30, 2 * R.scratch); }

// K panel of the residues of an operand of `rows` rows: the launch's, unless its residues take
// more than `limit` and than the operand's S BF16 slices would; then equal parts of it that do
// not (large build, 45 150 rows: 26 GB a panel in one part; cut in three, the contractions'
// passes over the results' residues made the build 9 % slower).
static int64_t residue_panel(int S, int n_mod, int64_t K, int64_t rows, int k_split, size_t limit)
{
    const int64_t kp = panel_k(K, rows, k_split);
    const size_t bytes = residue_bytes(n_mod, rows, kp);
    const size_t allowed = std::max(limit, residue_bytes(S, rows, kp));
    const int64_t parts = (int64_t)((bytes + allowed - 1) / allowed);
    return parts <= 1 ? kp : std::min(kp, ((kp + parts - 1) / parts + 511) / 512 * 512);
}

constexpr size_t kPanelBytes = (size_t)32 << 30;  // of one panel (and four limits) at most

static int64_t x_panel(const Request &R, int n_mod)
{
    return residue_panel(R.n_slices, n_mod, R.n2, n_pairs(R.nA), R.k_split,
                         std::min(kPanelBytes, 4 * R.scratch));
}

static bool p_resident(const Request &R, int n_mod, int64_t k_panel)
{
    return k_panel >= R.n2 || (size_t)((R.n2 + k_panel - 1) / k_panel) *
                                      residue_bytes(n_mod, n_pairs(R.nA), k_panel) <=
                                  resident_bytes(R);
}
static size_t p_bytes(const Request &R, int n_mod, int64_t k_panel)
{
    const int64_t panels = p_resident(R, n_mod, k_panel) ? (R.n2 + k_panel - 1) / k_panel : 1;
    return (size_t)panels * residue_bytes(n_mod, n_pairs(R.nA), k_panel);
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
    // residues of P (or of a K panel), the weighted AO values w chi_a on r2 they are formed
    // from, the int_2e operands' residues, and the residues of one pass of results
    const int n_mod = split_moduli(R.n_slices, std::max<int64_t>(R.n2, 3 * (int64_t)R.n1));
    const int64_t np = n_pairs(R.nA);
    size_t b = p_bytes(R, n_mod, x_panel(R, n_mod)) + 8 * (size_t)R.nA * R.n2 +
               std::min(min_residue_bytes(R), residue_bytes(n_mod, 4 * (int64_t)R.n1, R.n2)) +
               modular_out_bytes(n_mod, np,
                                 std::max<int64_t>(np, std::min<int64_t>(4 * (int64_t)R.n1, 1 << 30)),
                                 operand_bytes(R));
    if (!R.x_only)
        b += std::min(std::max(operand_bytes(R), residue_bytes(n_mod, np, 256)),
                      residue_bytes(n_mod, np, 3 * (int64_t)R.n1)) * 3;
    return b;
}

// The AO pairs (a, b) in the packed order of tri_index (a >= b) or stri_index (a > b).
__global__ void pairs_kernel(int nA, int strict, int2 *__restrict__ out)
{
    const int a = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
    if (a < nA && a >= b + strict)
        out[strict ? stri_index(a, b, nA) : tri_index(a, b, nA)] = make_int2(a, b);
}

static int make_pairs(Workspace &W, int slot, cudaStream_t st, int nA, bool strict, int2 **out)
{
    const int64_t n = strict ? n_strict_pairs(nA) : n_pairs(nA);
    void *p;
    CUTC_TRY(W.get(slot, std::max<size_t>(1, n) * sizeof(int2), &p));
    *out = (int2 *)p;
    if (n == 0)
        return CUTC_OK;
    pairs_kernel<<<dim3(ceil_div(nA, 128), nA), 128, 0, st>>>(nA, strict, *out);
    CUTC_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    return CUTC_OK;
}

// Row scales of an operand.
static int scale_slot(Workspace &W, int slot, int rows, int **sc)
{
    void *p;
    CUTC_TRY(W.get(slot, std::max<size_t>(1, rows) * sizeof(int), &p));
    *sc = (int *)p;
    return CUTC_OK;
}

// Where the residues of P's panel from k0 are (ax_whole).
static void *p_panel(const SplitPlan &sp, int n_mod, int np, int64_t k0)
{
    return (char *)sp.ax.p + (k0 / sp.k_panel) * residue_bytes(n_mod, np, sp.k_panel);
}

int split_prepare_x(Engine *E, const Request &R, cudaStream_t st, const double *wr2,
                    const double *aos2v, int64_t n1t, int slot0, SplitPlan &sp)
{
    Workspace &W = E->ws;
    sp.slot0 = slot0;
    sp.n1t = n1t;
    const int n_mod = sp.n_mod = split_moduli(R.n_slices, R.n2);
    const int np = (int)n_pairs(R.nA);
    void *p;
    CUTC_TRY(W.get(slot0 + SS_ERR, 64, &p));
    sp.err = (int *)p;
    CUTC_CUDA_TRY(cudaMemsetAsync(sp.err, 0, 4, st));
    CUTC_TRY(make_pairs(W, slot0 + SS_PAIRS_SYM, st, R.nA, false, &sp.pairs_sym));
    CUTC_TRY(make_pairs(W, slot0 + SS_PAIRS_ANTI, st, R.nA, true, &sp.pairs_anti));
    CUTC_TRY(scale_slot(W, slot0 + SS_AX_SC, np, &sp.sc_ax));
    CUTC_TRY(scale_slot(W, slot0 + SS_BX_SC, (int)(4 * n1t), &sp.sc_bx));
    sp.k_panel = x_panel(R, n_mod);
    CUTC_TRY(W.get(slot0 + SS_AX, p_bytes(R, n_mod, sp.k_panel), &p));
    sp.ax.p = p;
    sp.ax.rows = np;
    CUTC_TRY(W.get(slot0 + SS_WCHI2, std::max<size_t>(1, (size_t)R.nA * R.n2) * 8, &p));
    sp.wchi2 = (const double *)p;
    sp.aos2v = aos2v;
    sp.ax_whole = p_resident(R, n_mod, sp.k_panel);
    if (R.mol_tag && E->tag_x == R.mol_tag && E->tag_x_buf == sp.ax.p)
        return CUTC_OK;  // the same molecule's scales (and residues) are already there
    CUTC_TRY(weighted_aos(st, R.n2, R.nA, wr2, aos2v, (int64_t)R.n2, (double *)p));
    SrcSym src{sp.wchi2, aos2v, (int64_t)R.n2, (int64_t)R.n2, sp.pairs_sym};
    CUTC_TRY(row_scales(st, src, np, (int64_t)R.n2, sp.k_panel, n_mod, sp.sc_ax));
    if (sp.ax_whole)
        for (int64_t k0 = 0; k0 < R.n2; k0 += sp.k_panel) {
            const int64_t kp = std::min<int64_t>(sp.k_panel, R.n2 - k0);
            CUTC_TRY(residue_rows(st, n_mod, src, 0, np, R.n2, k0, kp, residue_pitch(kp), sp.sc_ax,
                                  p_panel(sp, n_mod, np, k0)));
        }
    E->tag_x = R.mol_tag;
    E->tag_x_buf = sp.ax.p;
    return CUTC_OK;
}

int split_x_tile(Engine *E, const Request &R, cudaStream_t st, SplitPlan &sp, const float2 *G,
                 int nb, double *Xb, int blk_rows, int ib, cudaEvent_t gemm_begin,
                 cudaEvent_t gemm_end)
{
    const int n_mod = sp.n_mod;
    const int64_t np = n_pairs(R.nA);
    SrcSym sa{sp.wchi2, sp.aos2v, (int64_t)R.n2, (int64_t)R.n2, sp.pairs_sym};
    SrcDenseDF sb{G, (int64_t)R.n2};
    CUTC_TRY(row_scales(st, sb, 4 * nb, (int64_t)R.n2, sp.k_panel, n_mod, sp.sc_bx));
    if (gemm_begin)
        CUTC_CUDA_TRY(cudaEventRecord(gemm_begin, st));
    // column (c, i) of the tile -> column c blk_rows + ib + i of the block
    const ModularOut out{Xb, np, nb, blk_rows, ib, 1.0, 0.0};
    CUTC_TRY(modular_contract(
        st, E->ws, sp.slot0 + SS_BX, sp.slot0 + SS_RES, x_residue_bytes(R, sp.n1t),
        operand_bytes(R), n_mod,
        (int)np, 4 * nb, R.n2, sp.k_panel, sp.ax, false, sp.sc_ax, sp.sc_bx, out, sp.err,
        [&](int, int, int64_t k0, int64_t kp, ResiduePlanes &a) -> int {
            if (sp.ax_whole) {
                a.p = p_panel(sp, n_mod, (int)np, k0);
                return CUTC_OK;
            }
            return residue_rows(st, n_mod, sa, 0, (int)np, R.n2, k0, kp, a.pitch, sp.sc_ax, a.p);
        },
        [&](int n0, int nc, int64_t k0, int64_t kp, const ResiduePlanes &b) {
            return residue_rows(st, n_mod, sb, n0, nc, R.n2, k0, kp, b.pitch, sp.sc_bx, b.p);
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
    const int64_t k3 = 3 * (int64_t)nb;
    const int n_mod = split_moduli(R.n_slices, k3);  // (of both contractions)
    const int64_t pan_h = int2e_panel_k(R, n_mod, nb, np);
    const int64_t pan_n = int2e_panel_k(R, n_mod, k3, np);
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
    const bool whole = modular_whole(n_mod, np, nb, pan_h, operand_bytes(R)) &&
                       modular_whole(n_mod, nl, k3, pan_n, operand_bytes(R)) &&
                       modular_pass_cols(n_mod, np, np, operand_bytes(R)) >= np;
    const bool keep_b = whole && nb == R.n1 && R.mol_tag && E->tag_i == R.mol_tag &&
                        E->tag_i_buf == sc_h;
    SrcSym s0{wchi, aos1, (int64_t)nb, ld1, sp.pairs_sym};
    SrcAnti sn{wchi, aos1, nb, nA, ld1, sp.pairs_anti};
    if (!keep_b) {
        CUTC_TRY(weighted_aos(st, nb, nA, wr1, aos1, ld1, wchi));
        CUTC_TRY(row_scales(st, s0, np, (int64_t)nb, pan_h, n_mod, sc_h));
        CUTC_TRY(row_scales(st, sn, nl, k3, pan_n, n_mod, sc_n));
    }
    const double beta = first ? 0.0 : 1.0;
    // Xt[(m nb + i) np + p]: X_3 is column block 3, X_012 the blocks 0..2
    const double *x3 = Xt + 3 * (int64_t)nb * np;
    CUTC_TRY(row_scales_cols(st, x3, np, np, nb, n_mod, sc_a));
    CUTC_TRY(modular_contract(
        st, W, slot0 + SS_BH, slot0 + SS_RES, operand_bytes(R), operand_bytes(R), n_mod, np, np, nb,
        pan_h, a, keep_b, sc_a, sc_h, ModularOut{H, np, np, 0, 0, 1.0, beta}, sp.err,
        [&](int, int, int64_t k0, int64_t kp, const ResiduePlanes &o) {
            return residue_cols(st, n_mod, x3, np, np, k0, kp, o.pitch, sc_a, o.p);
        },
        [&](int n0, int nc, int64_t k0, int64_t kp, const ResiduePlanes &o) {
            return residue_rows(st, n_mod, s0, n0, nc, nb, k0, kp, o.pitch, sc_h, o.p);
        }));
    if (nl > 0) {
        CUTC_TRY(row_scales_cols(st, Xt, np, np, k3, n_mod, sc_a));
        CUTC_TRY(modular_contract(
            st, W, slot0 + SS_BN, slot0 + SS_RES, operand_bytes(R), operand_bytes(R), n_mod, np, nl, k3,
            pan_n, a, keep_b, sc_a, sc_n, ModularOut{N, np, nl, 0, 0, -0.5, beta}, sp.err,
            [&](int, int, int64_t k0, int64_t kp, const ResiduePlanes &o) {
                return residue_cols(st, n_mod, Xt, np, np, k0, kp, o.pitch, sc_a, o.p);
            },
            [&](int n0, int nc, int64_t k0, int64_t kp, const ResiduePlanes &o) {
                return residue_rows(st, n_mod, sn, n0, nc, k3, k0, kp, o.pitch, sc_n, o.p);
            }));
    }
    E->tag_i = whole && nb == R.n1 ? R.mol_tag : 0;
    E->tag_i_buf = sc_h;
    return CUTC_OK;
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

// C = alpha A B^T of two sources through the split form, asynchronous on st; sp.err is set
// for split_check.
template <class Src>
static int gemm_sources(Engine *E, cudaStream_t st, int base, int n_slices, int M, int N,
                        int64_t K, Src sa, Src sb, double alpha, double *C, int64_t ldc,
                        SplitPlan &sp)
{
    Workspace &W = E->ws;
    const int n_mod = split_moduli(n_slices, K);
    const int64_t pan = residue_panel(n_slices, n_mod, K, M, 0, kPanelBytes);
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
    CUTC_TRY(row_scales(st, sa, M, K, pan, n_mod, sc_a));
    CUTC_TRY(row_scales(st, sb, N, K, pan, n_mod, sc_b));
    sp.err = err;
    return modular_contract(
        st, W, base + 4, base + 5, (size_t)8 << 30, (size_t)4 << 30, n_mod, M, N, K, pan, a, false, sc_a, sc_b,
        ModularOut{C, ldc, N, 0, 0, alpha, 0.0}, err,
        [&](int, int, int64_t k0, int64_t kp, const ResiduePlanes &o) {
            return residue_rows(st, n_mod, sa, 0, M, K, k0, kp, o.pitch, sc_a, o.p);
        },
        [&](int n0, int nc, int64_t k0, int64_t kp, const ResiduePlanes &o) {
            return residue_rows(st, n_mod, sb, n0, nc, K, k0, kp, o.pitch, sc_b, o.p);
        });
}

// Split-precision GEMM on device arrays: C[m + ldc n] = sum_k A[m K + k] B[n K + k].
int split_gemm_dense(Engine *E, cudaStream_t st, int n_slices, int M, int N, int64_t K,
                     const double *A, const double *B, double *C, int64_t ldc)
{
    SplitPlan sp;
    CUTC_TRY(gemm_sources(E, st, 200, n_slices, M, N, K, SrcDense{A, K}, SrcDense{B, K}, 1.0, C, ldc,
                          sp));
    return split_check(st, sp);
}

// C[m + ldc n] = alpha sum_k [A1 | A2][m, k] [B1 | B2][n, k] through the split form: the
// two products of the same output as ONE contraction over K1 + K2 (one row scale per row
// of the concatenation).  A1, B1 are K1-contiguous, A2, B2 K2-contiguous (device arrays);
// asynchronous on st (sp.err is set for split_check).
int split_gemm_concat(Engine *E, cudaStream_t st, int n_slices, int M, int N, int64_t K1,
                      const double *A1, const double *B1, int64_t K2, const double *A2,
                      const double *B2, double alpha, double *C, int64_t ldc, SplitPlan &sp)
{
    return gemm_sources(E, st, 210, n_slices, M, N, K1 + K2, SrcConcat{A1, A2, K1, K2},
                        SrcConcat{B1, B2, K1, K2}, alpha, C, ldc, sp);
}

}  // namespace cutc
