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
