"""The automatic design of a batch of small replicas (1,833 atoms on average):
phased up to 5 replicas and where there are fewer than 50 atoms per replica of
the batch on average, from 37 on here; graph branches between.  The replicas end
bit-identical to the same engines stepped alone on either side of each line."""
import numpy as np
import pytest

from rbmd_b200 import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replicas,phased", [(5, True), (6, False), (36, False), (37, True)])
def test_auto_design_follows_replica_count(cuda, rbx, replicas, phased):
    kinds = [systems.lj_electrolyte(n, seed=n) for n in (1000, 1200, 3300)]

    def engines():
        out = [rbx.Engine(kinds[k % 3], precision=rbx.MIXED, seed=5) for k in range(replicas)]
        for e in out:
            e.compute_forces(0)
        return out

    group = engines()
    batch = rbx.Batch(group)
    batch.step(6)
    assert batch.design == (rbx.Batch.PHASED if phased else rbx.Batch.BRANCHES)
    alone = [rbx.Engine(s, precision=rbx.MIXED, seed=5) for s in kinds]
    for e in alone:
        e.compute_forces(0)
        e.step(6)
    want = [e.get_state() for e in alone]
    for k, e in enumerate(group):
        got = e.get_state()
        for key in ("pos", "vel", "force"):
            assert np.array_equal(got[key], want[k % 3][key]), (k, key)
    batch.close()
    for e in group + alone:
        e.close()
