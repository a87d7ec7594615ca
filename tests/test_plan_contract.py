"""The plain form's contraction scratch in the device-memory plan (host arithmetic only)."""
import cutc_gb300 as cg


def test_plain_contraction_scratch_follows_the_budget():
    """The plain form's contraction scratch takes half of the tile budget at most (16 GiB
    where nothing limits it), beside P, H, N and what the pair terms keep."""
    n1, n2, nA, nN = 25000, 80000, 120, 10
    np_, nl = nA * (nA + 1) // 2, nA * (nA - 1) // 2
    own = 8 * (np_ * n2 + np_ * np_ + np_ * nl)
    fixed = [cg.plan(n1, n2, nA, nN, cg.PLAIN_FP64, device_pointers=True,
                     max_work_bytes=b)["fixed_bytes"] - own for b in (1 << 20, 1 << 30, 24 << 30)]
    assert fixed[0] < fixed[1] < fixed[2]
    assert fixed[2] - fixed[0] > 8 << 30
    # the rest: residues within 64 MiB (a tile's at least) and 512 MiB, scales, r2 terms
    pair = 1 << 30
    assert fixed[0] < (192 << 20) + pair and fixed[1] < (640 << 20) + pair


def test_split_contraction_scratch_follows_the_budget():
    """The split form likewise: under a small budget no more than P's K panels as 5 BF16
    slices (10 bytes an element), H, N and the smallest blocks; all of P's residues with a
    large one."""
    n1, n2, nA, nN = 25000, 80000, 120, 10
    np_, nl = nA * (nA + 1) // 2, nA * (nA - 1) // 2
    own = 8 * (np_ * np_ + np_ * nl)
    small, large = (cg.plan(n1, n2, nA, nN, cg.SPLIT_BF16, device_pointers=True,
                            max_work_bytes=b)["fixed_bytes"] - own for b in (1 << 20, 24 << 30))
    pair = 1 << 30
    assert small < 10 * np_ * 40000 + (1 << 30) + pair
    assert large > 26 * np_ * n2
