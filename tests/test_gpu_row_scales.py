"""Row scales of the modular contraction: the same digits for a row and the row times a power
of two, at any exponent, and digits that follow the row's 2-norm however long it is."""
import numpy as np
import pytest

import cutc_gb300 as cg

pytestmark = pytest.mark.gpu


def _split(A, B, S=5):
    import torch
    return cg.split_gemm_device(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(),
                                n_slices=S).cpu().numpy()


def _localised(rng, rows, K):
    """Rows whose values fall off by e every five columns from a centre of their own, to 1e-30."""
    c = rng.integers(0, K, size=rows)
    d = np.abs(np.arange(K)[None] - c[:, None]) / 5.0
    return rng.normal(size=(rows, K)) * np.exp(-np.minimum(d, 69.0))


@pytest.mark.parametrize("K", [40, 1000, 1500, 80000])
@pytest.mark.parametrize("localised", [False, True])
def test_rows_times_a_power_of_two(K, localised):
    rng = np.random.default_rng(K)
    make = _localised if localised else (lambda g, n, k: g.normal(size=(n, k)))
    A, B = make(rng, 9, K), rng.normal(size=(7, K))
    ref = _split(A, B)
    for e in (-60, -300, -950, 200, 900):
        assert np.array_equal(_split(A * 2.0 ** e, B), ref * 2.0 ** e), e


@pytest.mark.parametrize("K", [1000, 80000, (1 << 20) + 5])
@pytest.mark.parametrize("e", [0, -60])
def test_localised_rows_keep_their_digits(K, e):
    """Operands rounded at 2^-45 of their row norms: |error| <= 2^-45 (|a|_2 |b|_1 + |a|_1 |b|_2)."""
    rng = np.random.default_rng(K + 1)
    A, B = _localised(rng, 6, K), _localised(rng, 5, K)
    B[:3] = A[:3] * rng.uniform(0.5, 1.5, size=K)  # some that overlap
    got = _split(A * 2.0 ** e, B) / 2.0 ** e
    ref = (A.astype(np.longdouble) @ B.T.astype(np.longdouble)).astype(np.float64)
    n2, n1 = np.linalg.norm, lambda x, axis: np.abs(x).sum(axis)
    bound = n2(A, axis=1)[:, None] * n1(B, 1)[None] + n1(A, 1)[:, None] * n2(B, axis=1)[None]
    assert np.all(np.abs(got - ref) <= 2.0 ** -45 * bound + 2.0 ** -52 * np.abs(ref))
