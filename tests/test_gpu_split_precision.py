"""The split form's rounding against that of S 9-bit slices, which take a row to +-2^-9S of the
power of two above its maximum: dense rows, whose norm is far above their maximum, included.

The rounding errors of a row are spread evenly over at most that interval, so the root mean
square of the error of sum_k a_k b_k is at most
    sqrt((u_a^2 |b|^2 + u_b^2 |a|^2) / 3),   u = 2^-9S 2^ceil(log2 max),
and the result's own rounding to FP64 comes on top.
"""
import numpy as np
import pytest

import cutc_gb300 as cg

pytestmark = pytest.mark.gpu

ROWS = 40


@pytest.mark.parametrize("K", [1000, 16000, 80000])
@pytest.mark.parametrize("kind", ["normal", "even"])
def test_no_coarser_than_slices(K, kind):
    import torch
    rng = np.random.default_rng(K)
    if kind == "normal":
        A, B = rng.normal(size=(ROWS, K)), rng.normal(size=(ROWS, K))
    else:
        A, B = rng.uniform(0.5, 1.0, size=(ROWS, K)), rng.uniform(0.5, 1.0, size=(ROWS, K))
    ref = A.astype(np.longdouble) @ B.T.astype(np.longdouble)
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    top = lambda x: 2.0 ** np.ceil(np.log2(np.abs(x).max(axis=1)))  # noqa: E731
    na, nb = np.linalg.norm(A, axis=1), np.linalg.norm(B, axis=1)
    for S in (3, 4, 5, 6):
        err = np.asarray(cg.split_gemm_device(dA, dB, n_slices=S).cpu().numpy() - ref, dtype=np.float64)
        ua, ub = 2.0 ** (-9 * S) * top(A), 2.0 ** (-9 * S) * top(B)
        var = (ua[:, None] ** 2 * nb[None] ** 2 + ub[None] ** 2 * na[:, None] ** 2) / 3.0
        var = var + (2.0 ** -53 * np.abs(np.asarray(ref, dtype=np.float64))) ** 2 / 3.0
        # 1600 results: their mean square is within a tenth of its expectation
        assert np.mean(err ** 2 / var) < 1.1, (S, np.mean(err ** 2 / var))
