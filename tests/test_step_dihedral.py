"""CPU model of the dihedral kernels' step (``NQB_STEP5`` in
n_queens_b200/csrc/dfs_kernel.cuh, ``settle_level_dih`` at load): the count
step under the class rules, checked per task against the oracle's weighted
counts at every prefix depth of small boards."""
import numpy as np
import pytest

import oracle
from test_step_model import DihLanes, alive_columns, popc, sar1, shiftamt, shr_clamp

U = np.uint32


class CountingDihLanes(DihLanes):
    def __init__(self, N, c, l, r, cls, classes):
        super().__init__(N, c, l, r, cls, classes)
        row = popc(self.cols).astype(np.int64) - (32 - N)
        av, tie, w, wt = self.avail, self.tie_bit, self.w, self.w_tie
        at_last, at_n2 = (row >= N - 1) & (av != 0), (row == N - 2) & (av != 0)
        done = np.where(at_last, np.where(av & ~tie, w, wt), U(0))
        barred = np.where(at_n2, ~self.last_mask, U(0))
        alive = alive_columns(self.cols, self.ld | barred, self.rd, av)
        extra = np.where(((tie & ~self.cols) != 0) & ((alive & ~tie) != 0), wt - w, U(0))
        done = np.where(at_n2, popc(alive) * w + extra, done)
        self.credit += done.astype(np.uint64)
        self.avail = np.where(at_last | at_n2 | (av == 0), U(0), alive)
        self.rd = sar1(self.rd)

    def step(self):
        cols, ld, rd, avail = self.cols, self.ld, self.rd, self.avail
        bit = (U(0) - avail) & avail
        pb = bit != 0
        nc, nl, nr = cols + bit, ld + bit * U(2), (bit >> U(1)) + rd
        na = ~(nc | nl | nr)
        xl, xr = nl * U(2), sar1(nr)
        f0 = ~(nc | xl | xr)
        pc = popc(nc)
        p2 = (pc == 30) & pb
        barred = (pc > self.side_popc) & (~(nc | self.noside) != 0)
        na = np.where(barred, U(0), na)
        f0 = np.where(p2, f0 & self.last_mask, f0)
        ma = ((U(0) - f0) & f0) * U(0xFFFFFFFC)
        mb = shr_clamp(U(0x3FFFFFFF), shiftamt(f0))
        naf = na & (ma | mb)
        pd = (naf != 0) & pb & (~(nc | xl * U(2) | sar1(xr)) != 0)  # row N-2 is not kept out
        tie = p2 & ((self.tie_bit & ~nc) != 0) & ((naf & ~self.tie_bit) != 0)
        add = np.where(p2, popc(naf) * self.w, U(0)) + np.where(tie, self.w_tie - self.w, U(0))
        self.cnt += add.astype(np.uint64)
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


@pytest.mark.parametrize("N,k", [(N, k) for N in range(4, 9) for k in range(2, N - 1)] + [(9, 4), (10, 3), (10, 5)])
def test_weighted_counts(N, k):
    c, l, r, cls, classes = oracle.dihedral_expand(N, k)
    lanes = CountingDihLanes(N, c, l, r, cls, classes)
    got = lanes.run()
    np.testing.assert_array_equal(got, oracle.dihedral_count_tasks(N, k, c, l, r, cls))
    assert int(got.sum()) == oracle.total(N, 2)
    assert (lanes.deepest <= np.maximum(1, N - 1 - popc(np.ascontiguousarray(c, U)).astype(np.int64))).all()
