"""FP64 pair terms whose values are far below their operands' scales: r2 points close to a nucleus
whose terms all vanish there.  The error has to stay relative to the sum of the terms'
magnitudes, as that of the term by term sum."""
import numpy as np
import pytest

import cutc_gb300 as cg

pytestmark = pytest.mark.gpu


def _reference(r1, r2, rn, c, m, n, o):
    """grad1 u and the sums of the terms' magnitudes, (3, n1, n2) each, in long double."""
    ld = np.longdouble
    r1, r2, rn, c = (np.asarray(a, dtype=ld) for a in (r1, r2, rn, c))

    def scaled(d):
        r = np.sqrt((d * d).sum(-1))
        t = 1 / (1 + r)
        return r * t, (t * t / r)[..., None] * d

    f1, g1 = scaled(r1[:, None] - rn[None])
    f2, _ = scaled(r2[:, None] - rn[None])
    g, gg = scaled(r1[:, None] - r2[None])
    u = np.zeros((3,) + g.shape, dtype=ld)
    mag = np.zeros_like(u)
    for A in range(rn.shape[0]):
        for k in range(c.shape[1]):
            if abs(c[A, k]) < 1e-10:
                continue
            for x, y in ((m[A, k], n[A, k]), (n[A, k], m[A, k])):
                left = c[A, k] * x * f1[:, A] ** max(x - 1, 0)
                t = left[:, None] * (f2[:, A] ** y)[None] * g ** o[A, k]
                s = c[A, k] * o[A, k] * np.outer(f1[:, A] ** x, f2[:, A] ** y) * \
                    g ** max(o[A, k] - 1, 0)
                for d in range(3):
                    a, b = t * g1[:, A, d][:, None], s * gg[..., d]
                    u[d] += a + b
                    mag[d] += np.abs(a) + np.abs(b)
    return u, np.asarray(mag, dtype=np.float64)


def _run(r1, r2, rn, c, m, n, o):
    import torch
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (r1, r2, rn)]
    q = [torch.from_numpy(np.ascontiguousarray(a, dtype=t)).cuda()
         for a, t in ((c, np.float64), (m, np.int32), (n, np.int32), (o, np.int32))]
    G = torch.full((4, r1.shape[0], r2.shape[0]), float("nan"), dtype=torch.float64, device="cuda")
    assert cg.jast_bh_device(*d, *q, G) == cg.CUTC_OK
    return G.cpu().numpy()


@pytest.mark.parametrize("exps", ["even", "all"])
@pytest.mark.parametrize("n_nuc", [1, 3, 20])
@pytest.mark.parametrize("n1,n2", [(5, 70), (33, 257)])
def test_points_near_a_nucleus(exps, n_nuc, n1, n2):
    rng = np.random.default_rng(n_nuc + n2)
    rn = 2.5 * np.arange(n_nuc)[:, None] * np.array([[1.0, 0.3, 0.1]])
    r1 = rng.normal(size=(n1, 3)) * 1.5
    # r2 from 1 to 1e-6 around the first nucleus; every tenth point anywhere
    v = rng.normal(size=(n2, 3))
    r2 = v / np.linalg.norm(v, axis=1, keepdims=True) * 10.0 ** rng.uniform(-6, 0, size=(n2, 1))
    r2[::10] = rng.normal(size=r2[::10].shape) * 3.0
    terms = 6
    pool = np.array([2, 3, 4]) if exps == "even" else np.array([1, 2, 5, 6])
    c = np.zeros((n_nuc, terms))
    c[0] = rng.normal(size=terms)  # the other nuclei have no terms
    m, n = rng.choice(pool, size=(n_nuc, terms)), rng.choice(pool, size=(n_nuc, terms))
    o = rng.choice(np.array([0, 2, 3, 4]) if exps == "even" else np.arange(7), size=(n_nuc, terms))
    G = _run(r1, r2, rn, c, m, n, o)
    u, mag = _reference(r1, r2, rn, c, m, n, o)
    # a dozen roundings in a term, exponents up to 6 in its factors, twelve terms
    assert np.all(np.abs(np.asarray(G[:3] - u, dtype=np.float64)) <= 64 * 2.0 ** -53 * mag)
    lap = -0.5 * (G[0] ** 2 + G[1] ** 2 + G[2] ** 2)
    assert np.all(np.abs(G[3] - lap) <= 4 * 2.0 ** -53 * np.abs(lap))


def test_ordinary_points_as_before():
    """The general case beside it: every nucleus with terms of its own, r2 on a grid."""
    rng = np.random.default_rng(1)
    rn = rng.uniform(0, 4, size=(4, 3))
    r1, r2 = rng.normal(size=(20, 3)) * 2 + 2, rng.normal(size=(300, 3)) * 2 + 2
    c = rng.normal(size=(4, 9)) * 0.3
    m, n, o = (rng.choice(np.array([0, 2, 3, 4]), size=(4, 9)) for _ in range(3))
    G = _run(r1, r2, rn, c, m, n, o)
    u, mag = _reference(r1, r2, rn, c, m, n, o)
    assert np.all(np.abs(np.asarray(G[:3] - u, dtype=np.float64)) <= 64 * 2.0 ** -53 * mag)
