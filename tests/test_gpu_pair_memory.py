"""The pair terms alone with very many points on one side: scratch stays bounded, and the sub-tiles
and windows that this takes do not change a bit."""
import numpy as np
import pytest

import cutc_gb300 as cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2", [(300_000, 33), (3, 2_500_001)])
def test_many_points_on_one_side(n1, n2):
    import torch
    rng = np.random.default_rng(n1)
    nN, nB = 8, 6
    dev = [torch.from_numpy(a).cuda() for a in
           (rng.normal(size=(n1, 3)) * 3, rng.normal(size=(n2, 3)) * 3, rng.normal(size=(nN, 3)) * 3,
            rng.normal(size=(nN, nB)) * 0.3)] + \
          [torch.from_numpy(rng.integers(0, 7, size=(nN, nB)).astype(np.int32)).cuda() for _ in range(3)]
    r1, r2 = dev[:2]

    def run(a, b):
        G = torch.full((4, a.shape[0], b.shape[0]), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert cg.jast_bh_device(a, b, *dev[2:], G) == cg.CUTC_OK
        return G

    cg.load().cutc_release()
    G = torch.empty((4, n1, n2), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    assert cg.jast_bh_device(*dev, G) == cg.CUTC_OK
    # 2 GiB of either operand, the values of e-n terms and marks
    assert free0 - torch.cuda.mem_get_info()[0] < 5 << 30
    for sl in (slice(0, 20), slice(-20, None)):
        if n1 > n2:
            assert torch.equal(run(r1[sl].contiguous(), r2), G[:, sl])
        else:
            assert torch.equal(run(r1, r2[sl].contiguous()), G[:, :, sl])
