"""CPU model of the count step with its look-ahead (``NQB_STEP4`` in
n_queens_b200/csrc/dfs_kernel.cuh): the filtered step of test_step_model.py,
with the right diagonal pre-shifted too (a child's right mask is
(bit >> 1) + rd) and children above row N-2 dropped when the row two below them
has no free column.  Checked per task against the oracle on whole boards from
the smallest the step enters and on arbitrary 32-bit masks.  The node-count form
(``NQB_STEP4N``: the size of each child's unfiltered list instead of the
look-ahead, plus the root level's) is checked the same way."""
import numpy as np
import pytest

import oracle
from test_step_model import Lanes, need_slots, popc, sar1, shiftamt, shr_clamp


class LookAheadLanes(Lanes):
    def __init__(self, N, c, l, r, nodes=False):
        super().__init__(N, c, l, r)
        self.rd = sar1(self.rd)  # lane_rd<4>
        self.count_nodes = nodes
        last = np.uint32((1 << N) - 1)
        root = np.where((c & ~last) | (popc(c) >= N - 1), np.uint32(0), ~(c | l | r) & last)
        self.nodes = popc(root).astype(np.uint64)  # load_task's `placed`

    def step(self):
        one, two, mone, m4 = np.uint32(1), np.uint32(2), np.uint32(0xFFFFFFFF), np.uint32(0xFFFFFFFC)
        cols, ld, rd, avail = self.cols, self.ld, self.rd, self.avail
        bit = (avail * mone) & avail
        pb = bit != 0
        nc, nl, nr = bit * one + cols, bit * two + ld, (bit >> one) + rd
        na = ~(nc | nl | nr)
        xl, xr = nl * two, sar1(nr)
        f0 = ~(nc | xl | xr)
        ma = ((np.uint32(0) - f0) & f0) * m4
        mb = shr_clamp(np.uint32(0x3FFFFFFF), shiftamt(f0))
        pc = popc(nc)
        p2 = (pc == 30) & pb
        f1 = ~(nc | xl * two | sar1(xr))
        pg = (pc != 30) & pb
        if self.count_nodes:
            self.nodes += np.where(pb, popc(na), 0).astype(np.uint64)
        else:
            pg &= f1 != 0
        naf = na & (ma | mb)
        pd = (naf != 0) & pg
        self.cnt += np.where(p2, popc(naf), 0).astype(np.uint64)
        avail = avail ^ bit
        pk = (avail != 0) | pd
        idx = np.flatnonzero((avail != 0) & pd)
        self.stack[idx, self.sp[idx]] = np.stack([cols[idx], ld[idx], rd[idx], avail[idx]], axis=1)
        self.sp[idx] += 1
        self.deepest = np.maximum(self.deepest, self.sp)
        cols, ld, rd, avail = (np.where(pd, n, o) for n, o in ((nc, cols), (xl, ld), (xr, rd), (naf, avail)))
        idx = np.flatnonzero((self.sp != 0) & ~pk)
        self.sp[idx] -= 1
        cols[idx], ld[idx], rd[idx], avail[idx] = self.stack[idx, self.sp[idx]].T
        self.cols, self.ld, self.rd, self.avail = cols, ld, rd, avail


@pytest.mark.parametrize("N,k", [(4, 1), (5, 1), (6, 2), (7, 2), (8, 3), (10, 4), (11, 6)])
def test_whole_board_prefixes(N, k):
    c, l, r = oracle.expand(N, k)
    lanes = LookAheadLanes(N, c, l, r)
    np.testing.assert_array_equal(lanes.run(), oracle.count_tasks(N, c, l, r))
    assert (lanes.deepest <= need_slots(N, c)).all()


@pytest.mark.parametrize("N", [6, 9, 11])
def test_arbitrary_32bit_tasks(N):
    rng = np.random.default_rng(N)
    rand = lambda: rng.integers(0, 1 << 32, 2500, dtype=np.uint64).astype(np.uint32)
    c, l, r = rand() & rand() & rand() & np.uint32((1 << N) - 1), rand() & rand(), rand() & rand()
    got = LookAheadLanes(N, c, l, r).run()
    np.testing.assert_array_equal(got, oracle.count_tasks(N, c, l, r))
    assert got.sum() > 0


@pytest.mark.parametrize("N,k", [(4, 1), (5, 2), (7, 5), (8, 3), (8, 6), (10, 4)])
def test_node_counts(N, k):
    c, l, r = oracle.expand(N, k)
    lanes = LookAheadLanes(N, c, l, r, nodes=True)
    want, nodes = oracle.count_tasks(N, c, l, r, nodes=True)
    np.testing.assert_array_equal(lanes.run(), want)
    np.testing.assert_array_equal(lanes.nodes, nodes)
