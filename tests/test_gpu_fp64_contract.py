"""The plain form's FP64 contraction (modular products, DMMA below K = 16 and for operands
that are not finite) through cutc_x_ao_to_mo and cutc_no_2e, on integers whose products
and sums are exact in FP64: every element has to equal the plain sum.  K on both sides of
the rule (n_ao 15, 16, 17), columns at the edges of the 64, 128 and 256 wide tiles."""
import numpy as np
import pytest

import cutc_gb300 as cg

pytestmark = pytest.mark.gpu


def _ints(rng, *shape):
    return rng.integers(1, 100, size=shape).astype(np.float64) * rng.choice([-1.0, 1.0], size=shape)


def _mo(X, L, R):
    return np.einsum("mgbi,jb->jimg", np.einsum("mgba,ia->mgbi", X, L), R)


@pytest.mark.parametrize("n1,nA,n_mo", [(3, 15, 4), (7, 16, 64), (33, 17, 65), (5, 40, 129),
                                        (2, 20, 257), (600, 18, 3)])
@pytest.mark.parametrize("device", [False, True])
def test_x_ao_to_mo_is_exact_on_integers(n1, nA, n_mo, device):
    rng = np.random.default_rng(n1 + nA)
    X, L, R = _ints(rng, 3, n1, nA, nA), _ints(rng, n_mo, nA), _ints(rng, n_mo, nA)
    if device:
        import torch
        got = cg.x_ao_to_mo(*[torch.from_numpy(a).cuda() for a in (X, L, R)])
        torch.cuda.synchronize()
        got = got.cpu().numpy()
    else:
        got = cg.x_ao_to_mo(X, L, R)
    assert np.array_equal(got, _mo(X, L, R))


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_values_that_are_not_finite_propagate(bad):
    rng = np.random.default_rng(9)
    X, L, R = _ints(rng, 3, 40, 18, 18), _ints(rng, 5, 18), _ints(rng, 5, 18)
    X[1, 17, 4, 3] = bad
    with np.errstate(invalid="ignore"):
        ref = _mo(X, L, R)
    assert np.array_equal(cg.x_ao_to_mo(X, L, R), ref, equal_nan=True)


@pytest.mark.parametrize("n1", [5, 16, 400])
def test_no_2e_is_exact_on_integers(n1):
    rng = np.random.default_rng(n1)
    n = 11
    C1, X = _ints(rng, n * n, 3 * n1), _ints(rng, n * n, 3 * n1)
    C2, D2 = _ints(rng, n * n, n1), _ints(rng, n * n, n1)
    a = 0.5 * (C1 @ X.T + C2 @ D2.T)
    ref = (a + a.T).reshape(n, n, n, n).transpose(0, 2, 1, 3).reshape(n * n, n * n)
    assert np.array_equal(cg.no_2e(C1, X, C2, D2, n, n1), ref)
