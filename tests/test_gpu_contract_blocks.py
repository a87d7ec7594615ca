"""Plain builds under a small work budget: their contractions run in blocks of rows, K panels and
passes of columns, which change no bit of X and int_2e by no more than its blocks' sums."""
import numpy as np
import pytest

import cutc_gb300 as cg
from cutc_gb300 import synth

pytestmark = pytest.mark.gpu


def test_blocks_of_a_small_budget():
    # 2145 pairs: the residues of 512 columns take 79 MB, the limit's half is 32 MiB; a pass of
    # 256 columns takes 20 MB, its quarter is 16 MiB
    p = synth.make_problem(n_nuc=3, n_ao=65, n_grid1=700, n_grid2=1300, size_bh=5, seed=21)
    X, I = cg.build_integrals(p, cg.PLAIN_FP64)
    Xs, Is, st = cg.build_integrals(p, cg.PLAIN_FP64, max_work_bytes=48 << 20, with_stats=True)
    assert st["n_r1_tiles"] > 1
    assert np.array_equal(X, Xs)
    # int_2e: the blocks' shares are added in FP64
    assert np.abs(I - Is).max() <= 2e-15 * np.abs(I).max()


def test_check_of_many_panels():
    """cutc_no_2e under a budget that cuts K = 330 000 into 645 panels: the largest values of
    tmpC1 meet zeros, and every panel adds a little to the sums of magnitudes.  The error stays
    relative to sum |a b|."""
    import torch
    n_mo, n1 = 6, 110_000
    m2 = n_mo * n_mo
    rng = np.random.default_rng(12)
    C1, X = rng.normal(size=(m2, 3 * n1)), rng.normal(size=(m2, 3 * n1))
    C2, D2 = rng.normal(size=(m2, n1)), rng.normal(size=(m2, n1))
    C1[:, :3] *= 1e10
    X[:, :3] = 0.0
    dev = [torch.from_numpy(a).cuda() for a in (C1, X, C2, D2)]
    out = torch.empty((m2, m2), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    opt = cg.options(cg.PLAIN_FP64, device_pointers=True, max_work_bytes=1 << 20)
    import ctypes
    assert cg.load().cutc_no_2e(ctypes.byref(opt), n_mo, n1, *[t.data_ptr() for t in dev],
                                out.data_ptr()) == cg.CUTC_OK
    ld = np.longdouble

    def step(a):
        a = (a + a.T).reshape(n_mo, n_mo, n_mo, n_mo)
        return a.transpose(0, 2, 1, 3).reshape(m2, m2)

    ref = step(0.5 * (C1.astype(ld) @ X.T.astype(ld)) + 0.5 * (C2.astype(ld) @ D2.T.astype(ld)))
    mag = step(0.5 * (np.abs(C1) @ np.abs(X).T) + 0.5 * (np.abs(C2) @ np.abs(D2).T))
    err = np.abs(np.asarray(out.cpu().numpy() - ref, dtype=np.float64))
    assert np.all(err <= 4 * 2.0 ** -53 * mag), (err / mag).max() * 2.0 ** 53
