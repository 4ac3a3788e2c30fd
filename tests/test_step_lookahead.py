"""CPU models of the count steps with look-ahead (n_queens_b200/csrc/dfs_kernel.cuh),
operation by operation, checked per task against the oracle on whole boards from
the smallest the step enters and on arbitrary 32-bit masks:

* ``NQB_STEP4``: the filtered step of test_step_model.py with the right diagonal
  pre-shifted too (a child's right mask is (bit >> 1) + rd) and children above
  row N-2 dropped when the row two below them has no free column;
* ``NQB_STEP6``: the same in place -- the parent's remaining columns are pushed
  before the child is computed over it, and a child that is not entered is
  undone by a pop -- with one stack slot more;
* ``NQB_STEP7``: the same without the gate on row N-2 -- a counted child may be
  entered, finds no alive column and ends -- with a second extra slot;
* ``NQB_STEP6N``: its node-count form (the size of each child's unfiltered list
  instead of the look-ahead, plus the root level's)."""
import numpy as np
import pytest

import oracle
from test_step_model import Lanes, need_slots, popc, sar1, shiftamt, shr_clamp

ONE, TWO = np.uint32(1), np.uint32(2)


def alive_mask(f0):
    ma = ((np.uint32(0) - f0) & f0) * np.uint32(0xFFFFFFFC)
    return ma | shr_clamp(np.uint32(0x3FFFFFFF), shiftamt(f0))


class LookAheadLanes(Lanes):
    spared = 0

    def __init__(self, N, c, l, r, nodes=False):
        super().__init__(N, c, l, r)
        self.rd = sar1(self.rd)  # lane_rd
        self.count_nodes = nodes
        last = np.uint32((1 << N) - 1)
        root = np.where((c & ~last) | (popc(c) >= N - 1), np.uint32(0), ~(c | l | r) & last)
        self.nodes = popc(root).astype(np.uint64)  # load_task's `placed`

    def push(self, idx, cols, ld, rd, avail):
        self.stack[idx, self.sp[idx]] = np.stack([cols[idx], ld[idx], rd[idx], avail[idx]], axis=1)
        self.sp[idx] += 1
        self.deepest = np.maximum(self.deepest, self.sp)

    def step(self):
        cols, ld, rd, avail = self.cols, self.ld, self.rd, self.avail
        bit = (np.uint32(0) - avail) & avail
        pb = bit != 0
        nc, nl, nr = bit + cols, bit * TWO + ld, (bit >> ONE) + rd
        na = ~(nc | nl | nr)
        xl, xr = nl * TWO, sar1(nr)
        pc = popc(nc)
        p2 = (pc == 30) & pb
        pg = (pc != 30) & pb & (~(nc | xl * TWO | sar1(xr)) != 0)
        naf = na & alive_mask(~(nc | xl | xr))
        pd = (naf != 0) & pg
        self.cnt += np.where(p2, popc(naf), 0).astype(np.uint64)
        avail = avail ^ bit
        pk = (avail != 0) | pd
        self.push(np.flatnonzero((avail != 0) & pd), cols, ld, rd, avail)
        cols, ld, rd, avail = (np.where(pd, n, o) for n, o in ((nc, cols), (xl, ld), (xr, rd), (naf, avail)))
        idx = np.flatnonzero((self.sp != 0) & ~pk)
        self.sp[idx] -= 1
        cols[idx], ld[idx], rd[idx], avail[idx] = self.stack[idx, self.sp[idx]].T
        self.cols, self.ld, self.rd, self.avail = cols, ld, rd, avail


class InPlaceLanes(LookAheadLanes):
    spared = 1  # one slot more than need_slots
    gate = True

    def step(self):
        cols, ld, rd, avail = self.cols, self.ld, self.rd, self.avail
        bit = (np.uint32(0) - avail) & avail
        pb = bit != 0
        avail = avail ^ bit
        self.push(np.flatnonzero(avail), cols, ld, rd, avail)
        cols, ld, rd = cols + bit, ld + bit * TWO, rd + (bit >> ONE)
        na = ~(cols | ld | rd)
        ld, rd = ld * TWO, sar1(rd)
        f0 = ~(cols | ld | rd)
        pc = popc(cols)
        pg, p2 = ((pc != 30) | (not self.gate)) & pb, (pc == 30) & pb
        if self.count_nodes:
            self.nodes += np.where(pb, popc(na), 0).astype(np.uint64)
        else:
            pg &= ~(cols | ld * TWO | sar1(rd)) != 0
        avail = na & alive_mask(f0)
        pd = (avail != 0) & pg
        self.cnt += np.where(p2, popc(avail), 0).astype(np.uint64)
        avail = np.where(pd, avail, np.uint32(0))
        idx = np.flatnonzero((self.sp != 0) & ~pd)
        self.sp[idx] -= 1
        cols[idx], ld[idx], rd[idx], avail[idx] = self.stack[idx, self.sp[idx]].T
        self.cols, self.ld, self.rd, self.avail = cols, ld, rd, avail


class UngatedLanes(InPlaceLanes):
    spared = 2
    gate = False


@pytest.mark.parametrize("N,k", [(4, 1), (5, 1), (6, 2), (7, 2), (8, 3), (10, 4), (11, 6)])
@pytest.mark.parametrize("model", [LookAheadLanes, InPlaceLanes, UngatedLanes])
def test_whole_board_prefixes(N, k, model):
    c, l, r = oracle.expand(N, k)
    lanes = model(N, c, l, r)
    np.testing.assert_array_equal(lanes.run(), oracle.count_tasks(N, c, l, r))
    assert (lanes.deepest <= need_slots(N, c) + model.spared).all()


@pytest.mark.parametrize("N", [6, 9, 11])
@pytest.mark.parametrize("model", [LookAheadLanes, InPlaceLanes, UngatedLanes])
def test_arbitrary_32bit_tasks(N, model):
    rng = np.random.default_rng(N)
    rand = lambda: rng.integers(0, 1 << 32, 2500, dtype=np.uint64).astype(np.uint32)
    c, l, r = rand() & rand() & rand() & np.uint32((1 << N) - 1), rand() & rand(), rand() & rand()
    got = model(N, c, l, r).run()
    np.testing.assert_array_equal(got, oracle.count_tasks(N, c, l, r))
    assert got.sum() > 0


@pytest.mark.parametrize("N,k", [(4, 1), (5, 2), (7, 5), (8, 3), (8, 6), (10, 4)])
def test_node_counts(N, k):
    c, l, r = oracle.expand(N, k)
    lanes = InPlaceLanes(N, c, l, r, nodes=True)
    want, nodes = oracle.count_tasks(N, c, l, r, nodes=True)
    np.testing.assert_array_equal(lanes.run(), want)
    np.testing.assert_array_equal(lanes.nodes, nodes)
