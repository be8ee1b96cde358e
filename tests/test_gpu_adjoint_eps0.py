"""The force adjoint with LJ types of eps = 0 (sites without an LJ term)."""
import numpy as np
import pytest

from rbmd_b200 import systems

pytestmark = pytest.mark.gpu


def _vjp(rbx, s, prec, m):
    e = rbx.Engine(s, precision=prec)
    e.set_k_samples(*m)
    e.compute_forces(epoch=3)
    out = e.force_vjp(np.random.default_rng(6).normal(size=(s["n"], 3)))
    e.close()
    return out


@pytest.mark.parametrize("prec", [0, 1])
def test_unused_type_of_zero_eps(cuda, rbx, oracle, prec):
    """A type that no atom has contributes nothing: its gradients are 0, and
    every other gradient is what the system without it gives."""
    s = systems.lj_electrolyte(1500, seed=21)
    m = oracle.rbe_sample_philox(oracle.Box.make(s["lo"], s["hi"]), 0.16, 100, 3, 3)
    more = dict(s, sigma=np.append(s["sigma"], 1.0), eps=np.append(s["eps"], 0.0),
                mass=np.append(s["mass"], 1.0))
    want, got = _vjp(rbx, s, prec, m), _vjp(rbx, more, prec, m)
    assert got["eps"][3] == 0.0 and got["sigma"][3] == 0.0
    assert np.array_equal(got["eps"][:3], want["eps"])
    assert np.array_equal(got["sigma"][:3], want["sigma"])
    assert np.array_equal(got["pos"], want["pos"])


@pytest.mark.parametrize("prec", [0, 1])
def test_pairs_with_a_type_of_zero_eps(cuda, rbx, oracle, prec):
    """Water-like: one of the types has no LJ term.  Its own d_eps does not
    exist (NaN); every other gradient is finite and the FP64 adjoint's, at the
    tolerances of the adjoint's other comparisons (1e-9; FP32 terms 2e-5)."""
    from oracle import adjoint as A

    s = systems.lj_electrolyte(4000, seed=45)
    s["eps"] = np.array([1.3, 0.7, 0.0])
    p, n, ep = s["params"], s["n"], 3
    box, L = oracle.Box.make(s["lo"], s["hi"]), np.asarray(s["hi"]) - np.asarray(s["lo"])
    m = oracle.rbe_sample_philox(box, p["alpha"], p["kspace_p"], 3, ep)
    got = _vjp(rbx, s, prec, m)
    cols = lambda a: [np.ascontiguousarray(a[:, d]) for d in range(3)]  # noqa: E731
    perm, cell, cs, ce = oracle.cells_sort(box, 5.3, *cols(s["pos"]))
    pos = s["pos"][perm]
    cnt, rows = oracle.full_list(box, 5.3, *cols(pos), cell, cs, ce)
    freq = oracle.rbl_params(n, box, p["r_core"], p["cut_off"], p["neighbor_sample_num"])[0]
    cc, core, sc, shell = oracle.rbl_filter(box, p["r_core"], p["cut_off"], freq, ep,
                                            s["gid"][perm], *cols(pos), cnt, rows)
    g = np.random.default_rng(6).normal(size=(n, 3))
    with np.errstate(invalid="ignore"):
        d_eps, d_sig, d_q, d_alpha, d_r = A.force_vjp(
            pos, L, s["type"][perm], s["sigma"], s["eps"], s["q"][perm], p["alpha"], p["qqr2e"],
            p["r_core"], p["cut_off"], freq, A.rbl_pairs(cc, core, sc, shell, freq), m, g[perm])
    tol = 1e-9 if prec == 0 else 2e-5
    assert np.isnan(got["eps"][2]) and np.isnan(d_eps[2])
    assert np.abs(got["eps"][:2] - d_eps[:2]).max() <= tol * np.abs(d_eps[:2]).max()
    assert np.abs(got["sigma"] - d_sig).max() <= tol * np.abs(d_sig).max()
    assert abs(got["alpha"] - d_alpha) < tol * abs(d_alpha)
    assert systems.rel_rms(got["charge"][perm][:, None], d_q[:, None]) < tol
    assert systems.rel_rms(got["pos"][perm], d_r) < tol
