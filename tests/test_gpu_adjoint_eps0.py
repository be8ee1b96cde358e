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
