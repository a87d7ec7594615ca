"""FP64 contractions that accumulate (beta = 1) and take their columns in several passes, with
an operand that is not finite in a late column: the earlier columns are added once."""
import numpy as np
import pytest

import cutc_gb300 as cg

pytestmark = pytest.mark.gpu


def test_late_column_that_is_not_finite():
    """get_int_2e_ao with n_ao = 110: 12 100 x 12 100 results are more than one pass.  One
    AO's value and gradient of 1e200 at a point make S_m of that AO with itself, the last
    column, inf - inf; every element without that AO is finite and has to be right."""
    import torch
    nA, n1 = 110, 24
    rng = np.random.default_rng(3)
    w = rng.uniform(0.5, 1.5, n1)
    v = rng.normal(size=(4, nA, n1))
    v[0, nA - 1, 7] = v[1, nA - 1, 7] = 1e200
    Xh = rng.normal(size=(4, n1, nA, nA))
    dev = {k: torch.from_numpy(np.ascontiguousarray(a)).cuda()
           for k, a in dict(w=w, v=v, X=Xh).items()}
    I = torch.empty((nA * nA, nA * nA), dtype=torch.float64, device="cuda")
    cg.load().get_int_2e_ao(n1, nA, dev["w"].data_ptr(), dev["v"].data_ptr(),
                            dev["X"].data_ptr(), I.data_ptr())
    torch.cuda.synchronize()
    # the elements without the last AO, from its neighbours alone
    k = nA - 1
    got = I.view(nA, nA, nA, nA)[:k, :k, :k, :k].reshape(k * k, k * k)
    X = dev["X"][:, :, :k, :k].reshape(4, n1, k * k)
    c = dev["v"][0, :k]
    S0 = (c[:, None] * c[None] * dev["w"]).reshape(k * k, n1)  # [j + k i]: w chi_i chi_j
    A = S0 @ X[3]
    mag = S0.abs() @ X[3].abs()
    for m in range(3):
        d = dev["v"][1 + m, :k]
        S = (dev["w"] * (c[None] * d[:, None] - c[:, None] * d[None])).reshape(k * k, n1)
        A -= 0.5 * (S @ X[m])
        mag += 0.5 * (S.abs() @ X[m].abs())
    ref, mag = A + A.T, mag + mag.T
    # four sums of 24 products each, twice: below 256 roundings of the sum of magnitudes
    assert torch.all((got - ref).abs() <= 256 * 2.0 ** -53 * mag)
