"""The RBL filter, mean removal and row-wise state read-back at their edges:
rows that overflow either capacity, candidate counts around a warp's 64-entry
batch, rows that end at the largest 32-bit position, one atom, more atoms than
one block's partial sums.

Lists against a numpy restatement of the filter over the same candidates
(whole numbers, exactly); the mean removal against numpy in FP64 (1e-12; float
results to a float's 6e-8 of the largest force).
"""
import numpy as np
import pytest

from rbmd_b200 import systems

pytestmark = pytest.mark.gpu


def _mix(v):
    v = np.asarray(v, dtype=np.uint64) + np.uint64(0x9e3779b97f4a7c15)
    v = (v ^ (v >> np.uint64(30))) * np.uint64(0xbf58476d1ce4e5b9)
    v = (v ^ (v >> np.uint64(27))) * np.uint64(0x94d049bb133111eb)
    return v ^ (v >> np.uint64(31))


@pytest.mark.parametrize("freq", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("caps", [(128, 192), (7, 5), (0, 0)])
@pytest.mark.parametrize("lengths", [(0, 1, 31, 32, 63, 64, 65, 128, 200),
                                     (32, 0, 1, 7, 8, 15, 16, 17, 31)])  # all short
def test_filter_capacities(cuda, rbx, freq, caps, lengths):
    rng = np.random.default_rng(freq)
    n, L, epoch = 300, 20.0 if max(lengths) > 32 else 12.0, 9
    pos = rng.uniform(0, L, (n, 3))
    gid = rng.permutation(n).astype(np.int32) + 1
    # an atom may meet itself; the last rows are long again
    cand = [rng.choice(n, lengths[i % 9] if i < 290 else 70, replace=False) for i in range(n)]
    count = np.array([len(c) for c in cand])
    start = np.concatenate([[0], np.cumsum(count)[:-1]]).astype(np.int32)
    ccap, scap = caps
    core_start = (np.arange(n) * max(ccap, 1)).astype(np.int32)
    dev = lambda a: cuda.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    fill = lambda k: cuda.full((max(k, 1),), -1, dtype=cuda.int32, device="cuda")  # noqa: E731
    core_end, core, shell = fill(n), fill(n * ccap), fill(n * scap)
    snum, need, realloc = fill(n), dev(np.zeros(1, np.int32)), dev(np.zeros(1, np.int32))
    core2, force2 = 2.5 ** 2 - 1e-4, 25.0 - 1e-4
    rbx.rbl_filter(core2, force2, dev(gid), *(dev(pos[:, d]) for d in range(3)), dev(start),
                   dev((start + count).astype(np.int32)),
                   dev(np.concatenate(cand).astype(np.int32)),
                   dev(np.full(n, ccap, np.int32)), dev(core_start), core_end, core, scap, shell,
                   snum, need, rbx.Box.make([0] * 3, [L] * 3), realloc, freq, epoch)
    cuda.cuda.synchronize()
    a = _mix(gid.astype(np.uint64))
    with np.errstate(over="ignore"):
        b = _mix(gid.astype(np.uint64) + np.uint64(0xd1b54a32d192ed03))
        hcore, hshell = core.cpu().numpy(), shell.cpu().numpy().reshape(-1, n) if scap else None
        most_core = most = 0
        for i in range(n):
            j = cand[i][cand[i] != i]
            d = pos[i] - pos[j]
            d -= L * np.round(d / L)
            r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
            want_core = j[r2 < core2]
            hit = _mix(np.uint64(epoch) ^ a[i] ^ b[j]) % np.uint64(freq) == 0
            want = j[(r2 >= core2) & (r2 < force2) & hit]
            most_core, most = max(most_core, len(want_core)), max(most, len(want))
            c0, c1 = core_start[i], int(core_end[i])
            assert c1 - c0 == min(len(want_core), ccap)
            assert hcore[c0:c1].tolist() == want_core[:ccap].tolist()
            assert int(snum[i]) == min(len(want), scap)
            if scap:
                assert hshell[:int(snum[i]), i].tolist() == want[:scap].tolist()
    assert need.item() == most
    assert realloc.item() == (1 if most_core > ccap else 0)
    assert most_core > 0 and most > 0


@pytest.mark.parametrize("real", ["f64", "f32"])
def test_rows_at_the_last_positions(cuda, rbx, real):
    """A row that ends at INT_MAX gives what it gives elsewhere (filter, RBL and
    Verlet pair functors); its buffer holds 2^31 - 1 entries and no more."""
    t = cuda.float64 if real == "f64" else cuda.float32
    sfx = "" if real == "f64" else "_f32"
    rng = np.random.default_rng(2)
    n, L, k, end = 96, 6.0, 70, 2 ** 31 - 1
    dev = lambda a: cuda.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    ints = lambda *s: cuda.zeros(s, dtype=cuda.int32, device="cuda")  # noqa: E731
    g = np.stack(np.meshgrid(*[np.arange(5)] * 3), -1).reshape(-1, 3)[:n] * 1.2
    x = [dev((g[:, d] + rng.uniform(0, 0.1, n))).to(t) for d in range(3)]
    q, typ, gid = dev(rng.normal(size=n)).to(t), ints(n), dev(np.arange(n, dtype=np.int32))
    one, box = cuda.ones(1, dtype=t, device="cuda"), rbx.Box.make([0] * 3, [L] * 3)
    cand = rng.permutation(np.arange(1, n))[:k].astype(np.int32)
    buf = cuda.empty(end, dtype=cuda.int32, device="cuda")
    got = []
    for at in (0, end - k):  # atom 0's row; the other rows are empty
        buf[at:at + k] = dev(cand)
        start = ints(n) + at
        stop = start.clone()
        stop[0] = at + k
        core_start, core_end, core = ints(n), ints(n), ints(128)
        shell, snum, need, realloc = ints(64 * n), ints(n), ints(1), ints(1)
        getattr(rbx, "rbl_filter" + sfx)(2.0, 9.0, gid, *x, start, stop, buf, ints(n) + 128,
                                         core_start, core_end, core, 64, shell, snum, need, box,
                                         realloc, 2, 3)
        F, V = [cuda.zeros_like(q) for _ in range(3)], [cuda.zeros_like(q) for _ in range(3)]
        getattr(rbx, "pair_force_rbl" + sfx)(box, 2.0, 3.0, 10, 2, 0.16, 1.0, typ, one, one, start,
                                             stop, buf, shell, snum, q, *x, *F)
        vir, e = cuda.zeros(6 * n, dtype=t, device="cuda"), cuda.zeros(2, dtype=t, device="cuda")
        getattr(rbx, "pair_force_verlet" + sfx)(box, 3.0, 0.16, 1.0, typ, one, one, start, stop,
                                                buf, q, *x, *V, vir, e[:1], e[1:])
        cuda.cuda.synchronize()
        got.append([a.cpu().numpy() for a in (core_end, core, snum, shell, need, *F, *V, vir, e)])
    assert got[0][0][0] > 0 and got[0][2][0] > 0 and np.abs(got[0][8]).max() > 0
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [1, 255, 257, 148 * 256 + 3])
@pytest.mark.parametrize("real", ["f64", "f32"])
def test_mean_removal(cuda, rbx, n, real):
    rng = np.random.default_rng(n)
    t = cuda.float64 if real == "f64" else cuda.float32
    f = rng.normal(3.0, 20.0, (3, n)).astype(np.float64 if real == "f64" else np.float32)
    F = [cuda.as_tensor(v.copy()).cuda() for v in f]
    mean = cuda.zeros(3, dtype=t, device="cuda")
    (rbx.fix_rbl_force if real == "f64" else rbx.fix_rbl_force_f32)(*F, mean)
    cuda.cuda.synchronize()
    want_mean = f.astype(np.float64).mean(1)
    big, tol = np.abs(f).max(), 1e-12 if real == "f64" else 6e-8
    assert np.abs(mean.cpu().numpy() - want_mean).max() <= tol * big
    for d in range(3):
        want = f[d].astype(np.float64) - want_mean[d]
        assert np.abs(F[d].cpu().numpy() - want).max() <= 2 * tol * big


def test_state_rows_match_columns(cuda, rbx):
    """get_state (rows) against the column read-back of the C interface."""
    s = systems.lj_electrolyte(1500, seed=3)
    e = rbx.Engine(s, precision=rbx.MIXED)
    e.step(7)
    cols = [np.zeros(e.n) for _ in range(9)]
    rbx.check(rbx.lib().rbx_engine_get_state(e._h, *[rbx._np_ptr(c) for c in cols]), "get_state")
    st = e.get_state()
    for a, k in enumerate(("pos", "vel", "force")):
        assert st[k].shape == (e.n, 3) and st[k].flags.c_contiguous
        assert np.array_equal(st[k], np.stack(cols[3 * a:3 * a + 3], 1))
    v = np.full((e.n, 3), np.nan)
    rbx.check(rbx.lib().rbx_engine_get_state_rows(e._h, None, rbx._np_ptr(v), None), "rows")
    assert np.array_equal(v, st["vel"])
    e.close()
