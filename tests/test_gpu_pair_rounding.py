"""Rounding of the FP64 pair terms: the force of single pairs along x against 50
digits.  One rounding of a quotient or product is 0.43e-16 rms; the reference's
expression (two divisions) leaves 1.2e-16 of the larger LJ term and 1.3e-16 to
1.5e-16 of the Coulomb force, and the product with the distance adds one more:
1.3e-16 and 1.6e-16.  The bounds lie a quarter above; 1/r^2 cubed unrounded, or
1/r squared in its place, does not meet them (2.1e-16 and 1.8e-16).
"""
import mpmath as mp
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("term", ["lj", "coulomb"])
def test_rbl_functor_pair_rounding(cuda, rbx, term):
    rng = np.random.default_rng(3)
    k, L, rc, alpha = 3000, 40.0, 5.0, 0.16
    r = rng.uniform(0.9, 4.99, k)
    x = np.concatenate([np.zeros(k), r])  # atom i and its only neighbour i + k
    zero, n = np.zeros(2 * k), 2 * k
    sig = np.array([1.0, 1.13])
    eps = np.array([1.0, 0.7]) if term == "lj" else np.zeros(2)
    q = np.zeros(n) if term == "lj" else np.ones(n)
    typ = np.tile(np.arange(2), k).astype(np.int32)[np.argsort(np.arange(n) % k, kind="stable")]
    dev = lambda a: cuda.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    start = np.concatenate([np.arange(k), np.full(k, k)]).astype(np.int32)
    stop = np.concatenate([np.arange(1, k + 1), np.full(k, k)]).astype(np.int32)
    F = [dev(zero) for _ in range(3)]
    none = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    rbx.pair_force_rbl(rbx.Box.make([-1.0] * 3, [L] * 3), rc, rc, 1, 1, alpha, 1.0, dev(typ),
                       dev(sig), dev(eps), dev(start), dev(stop),
                       dev((np.arange(k) + k).astype(np.int32)), none, none, dev(q), dev(x),
                       dev(zero), dev(zero), *F)
    f = F[0].cpu().numpy()[:k]
    mp.mp.dps = 50
    err = []
    for i in range(k):
        d, ti, tj = mp.mpf(r[i]), typ[i], typ[i + k]
        d2 = mp.mpf(r[i] * r[i])
        if term == "lj":
            sg = mp.mpf((sig[ti] + sig[tj]) / 2)
            e = mp.sqrt(mp.mpf(eps[ti] * eps[tj]))
            u = sg ** 6 / d2 ** 3
            want, scale = -24 * e * (2 * u * u - u) / d2 * d, 24 * e * u / d2 * d * max(1, 2 * u)
        else:
            s, b = mp.sqrt(d2), mp.sqrt(mp.mpf(alpha))
            want = -(mp.erfc(b * s) / d2 + 2 * b * mp.exp(-mp.mpf(alpha) * d2) /
                     (mp.sqrt(mp.pi) * s)) / s * d
            scale = abs(want)
        err.append(float(abs(mp.mpf(f[i]) - want) / scale))
    rms = np.sqrt((np.array(err) ** 2).mean())
    print(term, rms)
    assert rms < (1.65e-16 if term == "lj" else 1.75e-16)
