"""FP64 contractions of subnormal operands, and results that are subnormal: what an FP64 sum
gives, with its rounding."""
import numpy as np
import pytest

import cutc_gb300 as cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,c", [(1e-310, 1e10),    # subnormal operand, normal results
                                 (1e-305, 1e-6),    # subnormal T and results
                                 (1e-322, 1e20)])   # a few bits each
def test_transform_of_subnormal_values(x, c):
    rng = np.random.default_rng(8)
    nA, n_mo, n1 = 20, 7, 33
    X = rng.normal(size=(3, n1, nA, nA)) * x
    L = rng.normal(size=(n_mo, nA)) * c
    R = rng.normal(size=(n_mo, nA))
    got = cg.x_ao_to_mo(X, L, R)
    # exact sums: scaled by powers of two into the normal range (T is rounded to a multiple of
    # 2^-1074 where it is subnormal)
    up = 2.0 ** 600
    T = np.einsum("mgba,ia->mgbi", X * up, L)
    ref = np.einsum("mgbi,jb->jimg", T, R) / up
    mag = np.einsum("mgbi,jb->jimg", np.einsum("mgba,ia->mgbi", np.abs(X) * up, np.abs(L)),
                    np.abs(R)) / up
    ulp = 2.0 ** -1074 * (1 + np.abs(R).sum(1))[:, None, None, None]
    assert np.all(np.abs(got - ref) <= 40 * 2.0 ** -53 * mag + ulp)
    assert np.count_nonzero(got) > 0.9 * got.size
