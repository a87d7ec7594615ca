"""FP64 contractions of rows that hardly overlap: the largest values of one operand meet zeros or
small values of the other.  The error has to stay relative to sum_k |a_k b_k|, as that of an FP64
sum, not to the rows' norms."""
import numpy as np
import pytest

import cutc_gb300 as cg

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _transform_check(X, L, R):
    """Both contractions of the transform against longer sums.  An FP64 sum of K terms is within
    K roundings of the sum of magnitudes; T and the result make it twice."""
    got = cg.x_ao_to_mo(X, L, R)
    ld = np.longdouble
    T = np.einsum("mgba,ia->mgbi", X.astype(ld), L.astype(ld))
    ref = np.einsum("mgbi,jb->jimg", T, R.astype(ld))
    mag = np.einsum("mgbi,jb->jimg", np.einsum("mgba,ia->mgbi", np.abs(X), np.abs(L)), np.abs(R))
    err = np.abs(np.asarray(got - ref, dtype=np.float64))
    # 8 roundings: well within what sums of 100 terms show, 2 sqrt(100) at most
    assert np.all(err <= 8 * EPS * mag), (err / np.where(mag > 0, mag, 1)).max() / EPS
    return got


@pytest.mark.parametrize("factor", [1e4, 1e8, 1e14, 1e30])
@pytest.mark.parametrize("mos", [1, 30])
@pytest.mark.parametrize("value", [0.0, 1e-12])
def test_orbitals_that_leave_out_large_aos(factor, mos, value):
    rng = np.random.default_rng(4)
    nA, n_mo, n1 = 100, 30, 5
    X = rng.normal(size=(3, n1, nA, nA))
    X[..., :10] *= factor
    X[..., :10, :] *= factor
    L, R = rng.normal(size=(n_mo, nA)), rng.normal(size=(n_mo, nA))
    L[:mos, :10] *= value / factor
    R[:mos, :10] *= value / factor
    _transform_check(X, L, R)


def test_graded_rows():
    rng = np.random.default_rng(6)
    nA, n_mo, n1 = 90, 31, 4
    X = rng.normal(size=(3, n1, nA, nA)) * 10.0 ** rng.uniform(-12, 12, size=(3, n1, nA, nA))
    L = rng.normal(size=(n_mo, nA)) * 10.0 ** rng.uniform(-12, 12, size=(n_mo, nA))
    _transform_check(X, L, L[::-1].copy())


def test_rows_without_overlap_are_zero():
    rng = np.random.default_rng(7)
    nA, n_mo = 64, 20
    X = rng.normal(size=(3, 3, nA, nA))
    X[..., 32:] = 0.0
    L = rng.normal(size=(n_mo, nA))
    L[:10, :32] = 0.0
    got = _transform_check(X, L, L)
    assert np.count_nonzero(got[:, :10]) == 0 and np.count_nonzero(got[:, 10:]) > 0


def test_int_2e_of_points_without_weight():
    """get_int_2e_ao (the operand with rows along the other axis): X is 1e10 and 1e20 at points
    whose weight is 0 and 1e-14."""
    import torch
    nA, n1 = 12, 60
    rng = np.random.default_rng(9)
    w, v = rng.uniform(0.5, 1.5, n1), rng.normal(size=(4, nA, n1))
    X = rng.normal(size=(4, n1, nA * nA))
    X[:, 20:25] *= 1e10
    w[20:25] = 0.0
    X[:, 40:42] *= 1e20
    w[40:42] = 1e-34
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (w, v, X)]
    I = torch.empty((nA * nA, nA * nA), dtype=torch.float64, device="cuda")
    cg.load().get_int_2e_ao(n1, nA, *[a.data_ptr() for a in d], I.data_ptr())
    torch.cuda.synchronize()
    c, ld = v[0], np.longdouble
    S0 = (c[:, None] * c[None] * w).reshape(nA * nA, n1)
    A = S0.astype(ld) @ X[3].astype(ld)
    mag = np.abs(S0) @ np.abs(X[3])
    for m in range(3):
        g = v[1 + m]
        p, q = c[None] * g[:, None] * w, c[:, None] * g[None] * w
        S = (p - q).reshape(nA * nA, n1)
        A -= 0.5 * (S.astype(ld) @ X[m].astype(ld))
        mag += 0.5 * ((np.abs(p) + np.abs(q)).reshape(nA * nA, n1) @ np.abs(X[m]))
    ref, mag = A + A.T, mag + mag.T
    # a few roundings in each S, and those of eight sums of 60 terms
    assert np.all(np.abs(np.asarray(I.cpu().numpy() - ref, dtype=np.float64)) <= 32 * EPS * mag)
