"""cutc_x_ao_to_mo keeps its scratch bounded however many AOs there are per MO, and the
blocks that this takes do not change a bit of the results."""
import pytest

import cutc_gb300 as cg

pytestmark = pytest.mark.gpu


def test_scratch_of_few_mos_from_many_aos():
    import torch
    nA, n_mo, n1 = 300, 10, 2000
    L = cg.load()
    L.cutc_release()
    gen = torch.Generator("cuda").manual_seed(2)

    def normal(*shape):
        return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=gen)

    X, cl, cr = normal(3, n1, nA, nA), normal(n_mo, nA), normal(n_mo, nA)
    out = torch.empty(n_mo, n_mo, 3, n1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    assert L.cutc_x_ao_to_mo(n1, nA, n_mo, 3, cl.data_ptr(), cr.data_ptr(), X.data_ptr(),
                             out.data_ptr(), 1, None) == cg.CUTC_OK
    torch.cuda.synchronize()
    # T (0.14 GB) and the contraction's blocks; the residues of all of X take 16 GB
    assert free0 - torch.cuda.mem_get_info()[0] < 9 << 30
    t = torch.einsum("mgba,ia->mgbi", X, cl)
    ref = torch.einsum("mgbi,jb->jimg", t, cr)
    # two sums of 300 terms: below 2 x 300 roundings of the sums of magnitudes
    mag = torch.einsum("mgbi,jb->jimg", torch.einsum("mgba,ia->mgbi", X.abs(), cl.abs()), cr.abs())
    assert torch.all((out - ref).abs() <= 600 * 2.0 ** -53 * mag)
    # a fifth of the points alone, in one block: the same bits
    part = X[:, :400].contiguous()
    few = torch.empty(n_mo, n_mo, 3, 400, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert L.cutc_x_ao_to_mo(400, nA, n_mo, 3, cl.data_ptr(), cr.data_ptr(), part.data_ptr(),
                             few.data_ptr(), 1, None) == cg.CUTC_OK
    torch.cuda.synchronize()
    assert torch.equal(few, out[..., :400])
