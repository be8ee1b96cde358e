"""The fused RBL kernel where its row segments end: near segments that hold
every candidate or almost none, far segments shorter than one 128-entry batch
or with every remainder of four, wide skins (most selected far pairs beyond
cut_off at the step), a box on which rows are a few entries long; both forms
against the oracle's RBL + RBE force (1e-9 / 1e-5 relative RMS, as the other
tests of this kernel: the sums' order differs, the pair set does not).
"""
import numpy as np
import pytest

from rbmd_b200 import systems

pytestmark = pytest.mark.gpu

# density, r_core, cut_off, skin, neighbor_sample_num
CASES = {
    "all_near": (0.8, 4.9, 5.0, 0.3, 100),
    "almost_all_far": (0.8, 0.9, 5.0, 0.3, 100),
    "wide_skin": (0.8, 2.5, 4.0, 1.5, 60),
    "short_rows": (0.02, 2.5, 5.0, 0.3, 2),
    "dilute": (0.01, 2.5, 5.0, 0.3, 2),
    "ragged_far": (0.3, 2.0, 4.4, 0.45, 20),
}


@pytest.mark.parametrize("name", list(CASES))
def test_rbl_segments(cuda, rbx, oracle, name):
    density, r_core, cut, skin, samples = CASES[name]
    s = systems.lj_electrolyte(4001, seed=77, density=density, r_core=r_core, cut_off=cut,
                               skin=skin, neighbor_sample_num=samples)
    box = oracle.Box.make(s["lo"], s["hi"])
    m = oracle.rbe_sample_philox(box, 0.16, 100, 5, 1)
    want = oracle.rbl_rbe_evaluation(s, m, epoch=3, pair_energy=False)
    for prec, tol in ((rbx.PLAIN_FP64, 1e-9), (rbx.MIXED, 1e-5)):
        e = rbx.Engine(s, precision=prec)
        e.set_k_samples(*m)
        e.compute_forces(epoch=3)
        assert e.stats().selection_frequency == want["freq"]
        f = e.get_state()["force"]
        assert systems.rel_rms(f, want["force"]) < tol, (prec, name)
        assert np.isfinite(f).all()
        e.close()


def test_dilute_steps_in_the_graph(cuda, rbx):
    """A box of two atoms a cell (its list is built by two launches): steps from
    the captured graph, rebuilds included, equal the launch-by-launch engine's."""
    s = systems.lj_electrolyte(3000, seed=8, density=0.01, temperature=40.0)
    out = []
    for graph in (True, False):
        e = rbx.Engine(s, precision=rbx.MIXED, seed=4)
        e.set_step_graph(graph)
        e.step(60)
        assert e.stats().rebuilds >= 2
        out.append(e.get_state())
        e.close()
    for k in ("pos", "vel", "force"):
        assert np.array_equal(out[0][k], out[1][k])
