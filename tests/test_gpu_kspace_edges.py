"""The k-space passes over charged atoms only: no charge at all, a few charged
atoms (threads share an atom's k-vectors), mostly charged tiles, all charged;
ragged atom and k counts, more k-vectors than one staged table.

Reference: direct FP64 sums in numpy over every atom.  FP64 tolerance: the
phase of |m| <= 40 turns carries 40 * 2^-53 * 2 pi = 3e-14 at most, amplified
by nothing in the sums, and a sum of N terms adds sqrt(N) 2^-53: 1e-12 covers
both.  Float: the coordinate's own rounding times |m|, 40 * 2^-24 = 2.4e-6 of
a turn, 1.5e-5 rad; the reference takes the same float coordinates, so only the
fixed-point step 2^-32 and the FP32 sine remain: 5e-6 as the golden tests use.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(257, 33, 0.0), (1000, 100, 0.03), (1003, 64, 0.4), (999, 129, 0.7), (512, 600, 1.0),
         (40001, 100, 0.1)]


def _system(n, p, share, seed):
    rng = np.random.default_rng(seed)
    lo, hi = np.array([0.0, 0.0, 0.0]), np.array([21.0, 18.5, 24.0])
    pos = rng.uniform(0, 1, (n, 3)) * (hi - lo)
    q = np.where(rng.uniform(size=n) < share, rng.choice([-1.0, 1.0, 0.5], n), 0.0)
    m = rng.integers(-12, 13, (3, p)).astype(float)
    m[0, (m == 0).all(0)] = 1.0
    return lo, hi, pos, q, m


def _direct(L, pos, q, m, S, p):
    k = 2 * np.pi * m / L[:, None]
    ph = pos @ k
    re, im = (q[:, None] * np.cos(ph)).sum(0), (q[:, None] * np.sin(ph)).sum(0)
    c = -4 * np.pi * S / (p * np.prod(L) * (k * k).sum(0))
    f = (c * (np.cos(ph) * im - np.sin(ph) * re)) @ k.T * q[:, None]
    return re, im, f


def _close(got, want, tol):
    scale = np.sqrt((want ** 2).mean())
    assert np.sqrt(((got - want) ** 2).mean()) <= tol * scale
    assert np.abs(got - want).max() <= 50 * tol * scale


@pytest.mark.parametrize("n,p,share", CASES)
@pytest.mark.parametrize("real", ["f64", "f32"])
def test_kspace_charged_shares(cuda, rbx, n, p, share, real):
    lo, hi, pos, q, m = _system(n, p, share, n + p)
    if real == "f32":
        pos, q = pos.astype(np.float32).astype(float), q.astype(np.float32).astype(float)
    L = hi - lo
    t = cuda.float64 if real == "f64" else cuda.float32
    dev = lambda a: cuda.as_tensor(np.ascontiguousarray(a)).to("cuda", t)  # noqa: E731
    box = rbx.Box.make(lo, hi)
    S = rbx.rbe_gauss_sum(box, 0.16)
    T = [dev(q), *(dev(v) for v in m), *(dev(pos[:, d]) for d in range(3))]
    rho = [cuda.zeros(p, dtype=t, device="cuda") for _ in range(2)]
    F = [cuda.full((n,), 7.0, dtype=t, device="cuda") for _ in range(3)]
    sf, fc = ((rbx.rbe_structure_factor, rbx.rbe_force) if real == "f64" else
              (rbx.rbe_structure_factor_f32, rbx.rbe_force_f32))
    sf(box, *T, *rho)
    fc(box, 0.16, S, 1.0, *rho, *T, *F)
    cuda.cuda.synchronize()
    re, im, f = _direct(L, pos, q, m, S, p)
    tol = 1e-12 if real == "f64" else 5e-6
    _close(np.stack([a.cpu().numpy() for a in rho]).astype(float), np.stack([re, im]), tol)
    got = np.stack([a.cpu().numpy() for a in F], 1).astype(float)
    _close(got, f, tol)
    assert (got[q == 0] == 0).all()


def test_kspace_fractional_k_and_far_positions(cuda, rbx):
    """The FP64 functors take any real k-vector and positions outside the box."""
    lo, hi, pos, q, m = _system(300, 40, 0.5, 3)
    m = m + 0.25
    pos = pos + 1000.0 * (hi - lo)
    L = hi - lo
    dev = lambda a: cuda.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    box = rbx.Box.make(lo, hi)
    T = [dev(q), *(dev(v) for v in m), *(dev(pos[:, d]) for d in range(3))]
    rho = [cuda.zeros(40, dtype=cuda.float64, device="cuda") for _ in range(2)]
    F = [cuda.zeros(300, dtype=cuda.float64, device="cuda") for _ in range(3)]
    rbx.rbe_structure_factor(box, *T, *rho)
    rbx.rbe_force(box, 0.16, 50.0, 1.0, *rho, *T, *F)
    cuda.cuda.synchronize()
    re, im, f = _direct(L, pos, q, m, 50.0, 40)
    # 36,750 turns at most: 36,750 * 2 pi * 2^-53 * 4 roundings = 1e-10
    _close(np.stack([a.cpu().numpy() for a in rho]), np.stack([re, im]), 1e-10)
    _close(np.stack([a.cpu().numpy() for a in F], 1), f, 1e-10)


def test_kspace_rounding(cuda, rbx):
    """Rounding of the FP64 functors beyond that of the phase k.r itself, which
    both sides form alike (k = 2 pi m / L, then fused multiply-adds): sine and
    cosine within an ulp and the sums' order, a few 2^-53 of the norm.  The
    reference takes the sines and sums in 80 bits.  (A phase from m and r / L,
    rounded otherwise, is 2.8e-15 away at this size.)"""
    rng = np.random.default_rng(4)
    n, p, L, S = 40000, 100, 36.84, 50.0
    pos, q = rng.uniform(0, L, (n, 3)), np.where(np.arange(n) % 4, 0.0, rng.choice([-1.0, 1.0], n))
    m = rng.integers(-9, 10, (3, p)).astype(float)
    m[0, (m == 0).all(0)] = 1.0
    ld = np.longdouble
    fma = lambda a, b, c: (ld(a) * ld(b) + ld(c)).astype(np.float64)  # noqa: E731
    k = 2 * np.pi * m / L
    c = -4 * np.pi * S / (p * L ** 3 * (k * k).sum(0))
    w = np.nonzero(q)[0]
    re, im, f = np.zeros(p), np.zeros(p), np.zeros((n, 3), dtype=ld)
    for a in range(p):
        ph = fma(k[2, a], pos[w, 2], fma(k[0, a], pos[w, 0], k[1, a] * pos[w, 1])).astype(ld)
        cs, sn = np.cos(ph), np.sin(ph)
        re[a], im[a] = (q[w] * cs).sum(), (q[w] * sn).sum()
        f[w] += (c[a] * (cs * im[a] - sn * re[a]) * q[w])[:, None] * k[:, a]
    dev = lambda a: cuda.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    box = rbx.Box.make([0] * 3, [L] * 3)
    T = [dev(q), *(dev(v) for v in m), *(dev(pos[:, d]) for d in range(3))]
    rho, F = [dev(np.zeros(p)) for _ in range(2)], [dev(np.zeros(n)) for _ in range(3)]
    rbx.rbe_structure_factor(box, *T, *rho)
    rbx.rbe_force(box, 0.16, S, 1.0, dev(re), dev(im), *T, *F)
    cuda.cuda.synchronize()
    err = lambda a, b: float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))  # noqa: E731
    assert err(np.stack([v.cpu().numpy() for v in rho]), np.stack([re, im])) < 8e-16
    assert err(np.stack([v.cpu().numpy() for v in F], 1), f) < 8e-16


@pytest.mark.parametrize("p", [7, 100, 1030])
def test_force_does_not_depend_on_the_block(cuda, rbx, p):
    """An atom's FP64 force is the same to the bit whatever shares its block:
    the charged atoms alone, among as many neutral atoms, and with 1 in 3, 6,
    12 and 40 charged (one to eight threads sum an atom's k-vectors)."""
    lo, hi, pos, _, m = _system(500, p, 1.0, p)
    q = np.random.default_rng(p).choice([-1.0, 0.5, 2.0], 500)
    rng = np.random.default_rng(1)
    dev = lambda a: cuda.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    box, rho = rbx.Box.make(lo, hi), [dev(rng.normal(size=p)) for _ in range(2)]
    ref = None
    for every in (1, 2, 3, 6, 12, 40):
        n = 500 * every
        at = np.sort(rng.choice(n, 500, replace=False))
        x, c = rng.uniform(0, 20, (n, 3)), np.zeros(n)
        x[at], c[at] = pos, q
        F = [dev(np.ones(n)) for _ in range(3)]
        rbx.rbe_force(box, 0.16, 50.0, 1.0, *rho, dev(c), *(dev(v) for v in m),
                      *(dev(x[:, d]) for d in range(3)), *F)
        f = np.stack([a.cpu().numpy() for a in F], 1)
        assert (np.delete(f, at, 0) == 0).all()
        ref = f[at] if ref is None else ref
        assert np.array_equal(f[at], ref), every


def test_kspace_any_phase(cuda, rbx):
    """Phases of 2^45 radians and far more still have a sine (positions are
    taken as they come)."""
    lo, hi, _, _, _ = _system(2, 1, 1.0, 0)
    L, mx = hi - lo, 3.0
    x = np.array([0.3, 1e13, -3e14, 7e15, 1e18, -1e30, 5e300])
    k = 2 * np.pi * mx / L[0]
    n, zero = len(x), np.zeros(len(x))
    dev = lambda a: cuda.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    m = [dev(np.array([v])) for v in (mx, 0.0, 0.0)]
    box = rbx.Box.make(lo, hi)
    for i in range(n):
        rho = [dev(np.zeros(1)) for _ in range(2)]
        rbx.rbe_structure_factor(box, dev(np.ones(1)), *m, dev(x[i:i + 1]), dev(zero[:1]),
                                 dev(zero[:1]), *rho)
        assert abs(rho[0].item() - np.cos(k * x[i])) < 4e-16
        assert abs(rho[1].item() - np.sin(k * x[i])) < 4e-16
    F = [dev(zero) for _ in range(3)]
    rbx.rbe_force(box, 0.16, 1.0, 1.0, dev(np.array([2.0])), dev(np.array([-1.0])),
                  dev(np.ones(n)), *m, dev(x), dev(zero), dev(zero), *F)
    c = -4 * np.pi / (np.prod(L) * k * k)
    want = c * (-np.cos(k * x) - 2.0 * np.sin(k * x)) * k
    assert np.abs(F[0].cpu().numpy() - want).max() < 1e-15 * abs(c * k) * 3


@pytest.mark.parametrize("n,kmax,share", [(300, (1, 1, 1), 1.0), (2000, (3, 2, 1), 0.1),
                                          (70, (0, 4, 2), 0.0),
                                          (2, (0, 0, 1), 1.0),  # one ion's force is rounding only
                                          (5000, (2, 3, 4), 0.5), (600, (11, 11, 11), 1.0)])
def test_ewald_blocks(cuda, rbx, oracle, n, kmax, share):
    lo, hi, pos, q, _ = _system(n, 1, share, n)
    dev = lambda a: cuda.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    cols = [np.ascontiguousarray(pos[:, d]) for d in range(3)]
    f, e = oracle.ewald_force(oracle.Box.make(lo, hi), 0.16, 1.0, list(kmax), q, *cols)
    F = [cuda.zeros(n, dtype=cuda.float64, device="cuda") for _ in range(3)]
    en = cuda.zeros(1, dtype=cuda.float64, device="cuda")
    rbx.ewald_force(rbx.Box.make(lo, hi), list(kmax), 0.16, 1.0, dev(q), *(dev(c) for c in cols),
                    *F, energy=en)
    cuda.cuda.synchronize()
    _close(np.stack([a.cpu().numpy() for a in F], 1), f, 1e-12)
    assert abs(en.item() - e) <= 1e-11 * abs(e)


@pytest.mark.parametrize("p", [1, 31, 256, 257, 1000])
def test_energy_virial_sums(cuda, rbx, p):
    """Energy and virial of given structure factors, FP64: sums of p terms."""
    lo, hi, _, _, m = _system(2, p, 1.0, p)
    L, V, alpha, S = hi - lo, float(np.prod(hi - lo)), 0.16, 40.0
    rng = np.random.default_rng(p)
    re, im = rng.normal(size=p), rng.normal(size=p)
    k = 2 * np.pi * m / L[:, None]
    k2 = (k * k).sum(0)
    base = 2 * np.pi * S / (p * V) * (re * re + im * im) / k2
    inner = 2 * (1 / (4 * alpha) + 1 / k2)
    vir = [(base * ((a == b) - inner * k[a] * k[b])).sum()
           for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
    e_self = np.sqrt(alpha / np.pi) * 3.0 + 0.5 * np.pi * 0.25 / (alpha * V)
    dev = lambda a: cuda.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    dv, de = dev(np.zeros(6)), dev(np.zeros(1))
    rbx.rbe_energy_virial(rbx.Box.make(lo, hi), alpha, S, 2.0, 3.0, 0.5, dev(re), dev(im),
                          *(dev(v) for v in m), dv, de)
    cuda.cuda.synchronize()
    scale = np.abs(base).sum()
    assert abs(de.item() - 2.0 * (base.sum() - e_self)) < 1e-13 * (scale + e_self)
    assert np.abs(dv.cpu().numpy() - 2.0 * np.array(vir)).max() < 1e-12 * np.abs(vir).max()
