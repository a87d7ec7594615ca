"""A device cutc_x_ao_to_mo returns while its work runs: plain calls on other streams, and
transforms on other streams, have to leave its scratch alone (and it theirs)."""
import numpy as np
import pytest

import cutc_gb300 as cg
from cutc_gb300 import synth

pytestmark = pytest.mark.gpu


def _transform(X, L, R, stream, out):
    n_mo, nA = L.shape
    s = cg.load().cutc_x_ao_to_mo(X.shape[1], nA, n_mo, X.shape[0], L.data_ptr(), R.data_ptr(),
                                  X.data_ptr(), out.data_ptr(), 1, stream.cuda_stream)
    assert s == cg.CUTC_OK


@pytest.mark.parametrize("other", ["build", "no_2e", "transform"])
def test_transform_beside_other_calls(other):
    import torch
    gen = torch.Generator("cuda").manual_seed(11)

    def normal(*shape):
        return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=gen)

    X, L, R = normal(3, 1501, 60, 60), normal(41, 60), normal(41, 60)
    out = torch.empty(41, 41, 3, 1501, dtype=torch.float64, device="cuda")
    X2, L2, R2 = normal(3, 700, 50, 50), normal(30, 50), normal(30, 50)
    out2 = torch.empty(30, 30, 3, 700, dtype=torch.float64, device="cuda")
    p = synth.make_problem(n_nuc=3, n_ao=14, n_grid1=300, n_grid2=900, size_bh=7, seed=5)
    C1, X4, C2, D2 = normal(196, 600), normal(196, 600), normal(196, 200), normal(196, 200)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def second():
        if other == "build":
            return cg.build_integrals(p, cg.PLAIN_FP64)[0]
        if other == "no_2e":
            return cg.no_2e(C1, X4, C2, D2, 14, 200).cpu().numpy()
        _transform(X2, L2, R2, b, out2)
        return out2

    _transform(X, L, R, a, out)
    torch.cuda.synchronize()
    ref = out.clone()
    ref2 = second()
    torch.cuda.synchronize()
    ref2 = ref2.clone() if other == "transform" else ref2
    for _ in range(10):
        out.fill_(float("nan"))
        torch.cuda.synchronize()
        _transform(X, L, R, a, out)
        got2 = second()
        torch.cuda.synchronize()
        assert torch.equal(out, ref)
        if other == "transform":
            assert torch.equal(got2, ref2)
        else:
            assert np.array_equal(got2, ref2)
