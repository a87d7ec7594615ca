"""The tensor-core pair terms: FP64 results and general exponents.

FP64 planes against the oracle within 1e-13 of each plane's largest value, the tolerance of
the other pair-kernel tests, for both coefficient layouts (exponents in {0, 2, 3, 4}; any up
to 6), at the edges of the 128-point r2 tiles and of the r1 groups of a tile (4 or 2 points),
at the largest nucleus counts of one contraction (16 and 9), one beyond, and three groups
of nuclei, with e-e and e-n coalescence.  The double-float form with general exponents, or
more nuclei than one contraction takes, against the oracle at the split form's tolerance and
against the double-float kernel at 1e-12."""
import numpy as np
import pytest

import cutc_gb300 as cg
from cutc_gb300 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu


def _problem(n_nuc, n1, n2, exps, seed, **kw):
    p = synth.make_problem(n_nuc=n_nuc, n_ao=5, n_grid1=n1, n_grid2=n2, size_bh=9, seed=seed,
                           box=1.5 + 0.4 * n_nuc, **kw)
    if exps == "all":
        rng = np.random.default_rng(seed)
        for f in ("m_bh", "n_bh", "o_bh"):
            setattr(p, f, rng.integers(0, 7, size=p.c_bh.shape).astype(np.int32))
    return p


@pytest.mark.parametrize("n1,n2", [(1, 127), (3, 128), (5, 129), (70, 1000)])
@pytest.mark.parametrize("n_nuc,exps", [(1, "even"), (16, "even"), (17, "even"), (40, "even"),
                                        (2, "all"), (9, "all"), (10, "all"), (20, "all")])
def test_fp64_planes_match_oracle(n1, n2, n_nuc, exps):
    import torch
    p = _problem(n_nuc, max(n1, n_nuc + 5), n2, exps, 50 + n_nuc)
    if n1 == 70:
        p = synth.add_coalescence(p)
    i0 = p.n_grid1 - n1
    d = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in p.arrays().items()}
    G = torch.full((4, n1, n2), float("nan"), dtype=torch.float64, device="cuda")
    s = cg.jast_bh_device(d["r1"], d["r2"], d["rn"], d["c_bh"], d["m_bh"], d["n_bh"], d["o_bh"], G,
                          i0=i0, n1b=n1, a_en=0.9, a_ee=1.2)
    assert s == cg.CUTC_OK, cg.last_error()
    p.a_en, p.a_ee = 0.9, 1.2
    ref = oracle.pair(p, i0, n1)
    got = G.cpu().numpy()
    scale = np.abs(ref).reshape(4, -1).max(axis=1)[:, None, None]
    assert np.all(np.abs(got - ref) <= 1e-13 * scale), np.max(np.abs(got - ref) / scale)


@pytest.mark.parametrize("n_nuc,exps", [(1, "all"), (12, "all"), (13, "all"), (25, "all"),
                                        (21, "even"), (40, "even")])
@pytest.mark.parametrize("slices", [5, 6])
def test_double_float_form_matches_its_kernel(monkeypatch, n_nuc, exps, slices):
    p = synth.add_coalescence(_problem(n_nuc, 130, 515, exps, 80 + n_nuc, a_en=1.1, a_ee=0.7))
    X1, I1 = cg.build_integrals(p, cg.SPLIT_BF16, n_slices=slices, x_components=4)
    monkeypatch.setenv("CUTC_PAIR_DF", "1")
    X2, I2 = cg.build_integrals(p, cg.SPLIT_BF16, n_slices=slices, x_components=4)
    assert oracle.rel_err(X1, X2)["max"] < 1e-12 and oracle.rel_err(I1, I2)["max"] < 1e-12
    Xo, Io = oracle.cutc_int(p)
    assert oracle.rel_err(X1[:3], Xo)["max"] < 1e-10 and oracle.rel_err(I1, Io)["max"] < 1e-10
