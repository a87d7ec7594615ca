"""Pair terms of split builds with general exponents and with many nuclei, where they are far below
their operands' scales: r2 close to a nucleus whose terms all vanish there.  With one r2 point X
is w chi_a chi_b grad1 u of that point, rounded at 2^-45 by the contraction's operands."""
import numpy as np
import pytest

import cutc_gb300 as cg
from cutc_gb300 import synth
from test_gpu_pair_precision import _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_nuc,exps", [(1, "all"), (2, "all"), (12, "all"), (24, "even")])
@pytest.mark.parametrize("distance", [1e-4, 0.02, 0.3, 2.0])
def test_point_near_a_nucleus(n_nuc, exps, distance):
    rng = np.random.default_rng(n_nuc)
    p = synth.make_problem(n_nuc=n_nuc, n_ao=2, n_grid1=60, n_grid2=1, size_bh=6, seed=3)
    pool = np.array([2, 3, 4]) if exps == "even" else np.array([1, 2, 5, 6])
    p.c_bh = np.zeros((n_nuc, 6))
    p.c_bh[0] = rng.normal(size=6)  # the other nuclei have no terms
    p.m_bh, p.n_bh = (rng.choice(pool, size=(n_nuc, 6)).astype(np.int32) for _ in range(2))
    p.o_bh = rng.choice(np.array([0, 2, 3, 4]), size=(n_nuc, 6)).astype(np.int32)
    p.r2 = p.rn[:1] + distance * np.array([[0.6, 0.0, 0.8]])
    p.wr2 = np.ones(1)
    p.aos2 = np.ones((4, 2, 1))
    p.r1 = np.ascontiguousarray(p.rn[0] + rng.normal(size=(60, 3)) * 1.5)
    X = cg.build_integrals(p, cg.SPLIT_BF16, 5)[0][:, :, 0]
    u, mag = _reference(p.r1, p.r2, p.rn, p.c_bh, p.m_bh, p.n_bh, p.o_bh)
    err = np.abs(np.asarray(X - u[:, :, 0], dtype=np.float64))
    # double-float terms (2^-44 of their magnitudes, six terms) and two roundings at 2^-45
    assert np.all(err <= 2.0 ** -43 * mag[:, :, 0]), (err / mag[:, :, 0]).max() * 2.0 ** 43
