"""FP64 pair terms of the largest number of nuclei, with coefficients of one size and sign and all
distances large: the largest sums over the nuclei that the integer accumulation can meet."""
import numpy as np
import pytest

from test_gpu_pair_precision import _reference, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exps", ["even", "all"])
def test_largest_sums(exps):
    n_nuc = 128
    rng = np.random.default_rng(3)
    rn = rng.uniform(-1, 1, size=(n_nuc, 3))
    v = rng.normal(size=(16, 3))
    r1 = v / np.linalg.norm(v, axis=1, keepdims=True) * rng.uniform(50, 1e6, size=(16, 1))
    v = rng.normal(size=(80, 3))
    r2 = v / np.linalg.norm(v, axis=1, keepdims=True) * rng.uniform(1e3, 1e6, size=(80, 1))
    pairs = [(x, y) for x in (0, 2, 3, 4) for y in (0, 2, 3, 4)] if exps == "even" else \
        [(x, y) for x in range(7) for y in range(7)]
    m, n = (np.array([p[k] for p in pairs * 1])[None].repeat(n_nuc, 0) for k in (0, 1))
    m, n = m[:, :32], n[:, :32]
    o = np.full_like(m, 2)
    c = np.full(m.shape, 0.999)
    G = _run(r1, r2, rn, c, m, n, o)
    u, mag = _reference(r1, r2, rn, c, m, n, o)
    # 64 to 128 nuclei times 32 terms of one sign: within 2 sqrt(8192) roundings
    assert np.all(np.abs(np.asarray(G[:3] - u, dtype=np.float64)) <= 180 * 2.0 ** -53 * mag)
