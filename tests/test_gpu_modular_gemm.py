"""The modular contraction (residue products on tcgen05 CTA pairs) on integer operands.

Integers up to 2^12 keep every bit on the row scales (an operand's scaled integers lie
2^-45 of its row norm apart) and every product sum is below 2^53, so the result is exact:
each element has to equal the integer product.  Sizes at the edges of the 256 x 256 and
256 x 128 tiles, of the 64-wide K blocks and of the 512-wide chunks; constant rows give
every product of a chunk the same residues, the largest sums a chunk can have.
"""
import numpy as np
import pytest

import cutc_gb300 as cg

pytestmark = pytest.mark.gpu


def _split(A, B, S=5):
    import torch
    return cg.split_gemm_device(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(),
                                n_slices=S).cpu().numpy()


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (256, 256, 64), (257, 129, 65), (255, 128, 511),
                                   (128, 257, 512), (300, 1025, 513), (2049, 2100, 1100),
                                   (9, 5, 70000)])
@pytest.mark.parametrize("S", [5, 7])
def test_integer_products_are_exact(M, N, K, S):
    rng = np.random.default_rng(M + N + K)
    A = rng.integers(-4096, 4097, size=(M, K)).astype(np.float64)
    B = rng.integers(-4096, 4097, size=(N, K)).astype(np.float64)
    assert np.array_equal(_split(A, B, S), A @ B.T)


@pytest.mark.parametrize("K", [511, 512, 1536])
def test_constant_rows_are_exact(K):
    """Every residue of a row equal: 40 values reach the ends of the residue range."""
    a = np.arange(1, 41, dtype=np.float64) * 101.0
    A = np.repeat(a[:, None], K, axis=1)
    assert np.array_equal(_split(A, -A), -(A @ A.T))


def test_rows_that_are_not_finite():
    """An infinity or a NaN makes its row's (column's) results NaN and no others."""
    rng = np.random.default_rng(5)
    A = rng.integers(-99, 100, size=(130, 200)).astype(np.float64)
    B = rng.integers(-99, 100, size=(70, 200)).astype(np.float64)
    R = A @ B.T
    A[3, 7], B[5, 199] = np.nan, np.inf
    C = _split(A, B)
    bad = np.zeros_like(R, dtype=bool)
    bad[3], bad[:, 5] = True, True
    assert np.all(np.isnan(C[bad])) and np.array_equal(C[~bad], R[~bad])


def test_products_of_several_streams():
    """Builds of different sizes on four streams at a time: the CTA pairs of one stream start
    and end beside the kernels of the others, and every result stays the same."""
    from cutc_gb300 import synth
    ps = [synth.make_problem(nn, na, 250 * nn, 1000 * nn, 9, 40 + nn)
          for nn, na in ((2, 52), (8, 10), (3, 30))]
    srv = cg.Server(n_slots=4, device_budget_bytes=32 << 30, cache_budget_bytes=1 << 30,
                    tile_budget_bytes=1 << 30)
    try:
        first = None
        for _ in range(200):
            tickets = [srv.submit(p, k + 1, cg.SPLIT_BF16, 5) for k, p in enumerate(ps + ps[:1])]
            out = [[a.copy() for a in srv.wait(t)[:2]] for t in tickets]
            first = first or out
            for got, ref in zip(out, first):
                assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
    finally:
        srv.close()
