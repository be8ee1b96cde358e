"""The stencil list builder where its tiles end: groups and chunks with
remainders, cells of several cull words, more surviving chunks than one
staged batch, more cull words than one pass, cells with one atom or none, dense
cells in a mostly empty box (whose cells of few atoms take other blocks), an
orthorhombic box away from the origin.

Rows must equal, in order, the FP64 predicate (minimum image, squares summed
left to right) over the 27 stencil cells in stencil order and the atoms of a
cell in cell order; whole numbers, so exactly.  A random subset of the atoms
is restated in numpy.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _uniform(n, lo, hi, seed):
    rng = np.random.default_rng(seed)
    lo, hi = np.asarray(lo, float), np.asarray(hi, float)
    return lo, hi, lo + rng.uniform(0.0, 1.0, (n, 3)) * (hi - lo)


def _clusters(per_cell, seed, side=3.0):
    """27 unit cells, each with per_cell atoms within 0.004 of its centre, in a
    box of side^3 such cells."""
    rng = np.random.default_rng(seed)
    k = np.arange(27)
    cen = np.stack([k % 3, (k // 3) % 3, k // 9], 1) + 0.5
    pos = np.repeat(cen, per_cell, 0) + rng.uniform(-0.002, 0.002, (27 * per_cell, 3))
    return np.zeros(3), np.full(3, side), pos


def _gas_and_drops(seed):
    """Clusters of 300 atoms in one corner of 16^3 cells, every other cell with
    none to a dozen atoms."""
    lo, hi, pos = _clusters(300, seed, 16.0)
    rng = np.random.default_rng(seed + 1)
    gas = rng.uniform(0.0, 16.0, (4000, 3))
    near = rng.uniform(0.0, 4.0, (200, 3)) + 6.0
    return lo, hi, np.concatenate([pos, gas, near])


CASES = {
    "three_cells_n3300": (lambda: _uniform(3300, [0] * 3, [16.1] * 3, 1), 5.3),
    "full_cells": (lambda: _uniform(27000, [0] * 3, [3.0] * 3, 8), 0.99),
    "dense_batches": (lambda: _uniform(20000, [0] * 3, [12.0] * 3, 2), 3.0),
    "many_cull_words": (lambda: _clusters(1300, 3), 0.99),
    "gas_and_drops": (lambda: _gas_and_drops(7), 0.99),
    "drops_in_a_void": (lambda: _clusters(1300, 3, 24.0), 0.99),
    "sparse_n40": (lambda: _uniform(40, [0] * 3, [30.0] * 3, 4), 5.0),
    "orthorhombic_offset": (lambda: _uniform(5003, [-7, 3, 100], [13, 20, 123], 5), 4.1),
}


@pytest.mark.parametrize("name", list(CASES))
def test_list_rows_in_order(cuda, rbx, name):
    (lo, hi, pos), rc = CASES[name][0](), CASES[name][1]
    n, L = len(pos), hi - lo
    box = rbx.Box.make(lo, hi)
    dims = rbx.cell_grid(box, rc)
    ncell = int(np.prod(dims))
    dev = lambda a: cuda.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    ints = lambda *s: cuda.zeros(s, dtype=cuda.int32, device="cuda")  # noqa: E731
    perm, cell, start = ints(n), ints(n), ints(ncell + 1)
    scratch = cuda.zeros(rbx.cells_scratch_bytes(n, ncell), dtype=cuda.uint8, device="cuda")
    rbx.cells_sort(box, rc, *[dev(pos[:, d]) for d in range(3)], perm, cell, start, scratch)
    order = perm.cpu().numpy()
    p, c, cs = pos[order], cell.cpu().numpy(), start.cpu().numpy()

    def row(i):
        cx, cy, cz = c[i] % dims[0], (c[i] // dims[0]) % dims[1], c[i] // (dims[0] * dims[1])
        out = []
        for s in range(27):
            k = [(cx + s % 3 - 1) % dims[0], (cy + (s // 3) % 3 - 1) % dims[1],
                 (cz + s // 9 - 1) % dims[2]]
            q = (k[2] * dims[1] + k[1]) * dims[0] + k[0]
            j = np.arange(cs[q], cs[q + 1])
            d = p[i] - p[j]
            d = np.where(np.abs(d) > 0.5 * L, d - np.where(d > 0, L, -L), d)
            r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
            out.append(j[(r2 < rc * rc) & (j != i)])
        return np.concatenate(out)

    pick = np.random.default_rng(9).choice(n, min(n, 200), replace=False)
    want = {int(i): row(i) for i in pick}
    count, overflow = ints(n), ints(1)
    xs = [dev(p[:, d]) for d in range(3)]
    rbx.full_list(box, rc, *xs, start, 1, count, ints(n, 1), overflow)  # counts; rows overflow
    cap = max(int(count.max()), 1)
    overflow.zero_()
    rows = cuda.full((n, cap), -1, dtype=cuda.int32, device="cuda")
    rbx.full_list(box, rc, *xs, start, cap, count, rows, overflow)
    cuda.cuda.synchronize()
    assert overflow.item() == 0
    got, cnt = rows.cpu().numpy(), count.cpu().numpy()
    for i, w in want.items():
        assert cnt[i] == len(w)
        assert np.array_equal(got[i, :cnt[i]], w)
        assert (got[i, cnt[i]:] == -1).all()
