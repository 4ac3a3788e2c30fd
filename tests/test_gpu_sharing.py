"""Shares of tasks and the mailbox between warps, on the GPU: every count against
the oracle where few tasks meet many lanes, at the list lengths where the
dealing changes, and where one task holds nearly all the work."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


# N=12: too few rows for the mailbox; N=15, k=1..2: 13 and 14 rows left, used.
@pytest.mark.parametrize("N,k", [(12, 3), (15, 1), (15, 2)])
def test_few_tasks_per_task_counts_and_nodes(gpu, N, k):
    c, l, r = oracle.expand(N, k)
    cnt, nodes = oracle.count_tasks(N, c, l, r, nodes=True)
    got = gpu.count_tasks(N, c, l, r, per_task=True, nodes=True)
    assert np.array_equal(got["per_task"], cnt) and np.array_equal(got["nodes"], nodes)
    got = gpu.count_tasks(N, c, l, r, per_task=True)
    assert np.array_equal(got["per_task"], cnt) and got["sum"] == int(cnt.sum())
    assert gpu.count_tasks(N, c, l, r)["sum"] == int(cnt.sum())
    for cfg in (dict(steal=-1), dict(block_threads=32, blocks_per_sm=1), dict(inner_steps=16), dict(layout=1)):
        assert gpu.count_tasks(N, c, l, r, config=cfg)["sum"] == int(cnt.sum()), cfg


# lanes = 148 SMs x 64 threads: the list lengths around 1/16, 1/8, 1, 4 and 8
# tasks per lane and around the finely dealt end of the queue.
@pytest.mark.parametrize("n", [1, 31, 591, 593, 1183, 1185, 2367, 2369, 9471, 9473, 37889, 75775, 75777])
def test_list_lengths(gpu, n):
    N, k = 14, 6
    c, l, r = (np.resize(a, n) for a in oracle.expand(N, k))
    base = oracle.count_tasks(N, *oracle.expand(N, k))
    want = np.resize(base, n)
    cfg = dict(block_threads=64, blocks_per_sm=1)
    got = gpu.count_tasks(N, c, l, r, per_task=True, config=cfg)
    assert np.array_equal(got["per_task"], want)
    q = max(1, n - n // 3)
    assert gpu.count_tasks(N, c, l, r, config=dict(cfg, queue_len=q))["sum"] == int(want[:q].sum())


def test_one_heavy_task_among_finished_ones(gpu):
    # One empty N=16 board and 20,000 boards without a free column: the heavy
    # task has to spread over the grid, again and again on the same scratch.
    n = 20000
    c = np.full(n, (1 << 15) - 1, np.uint32)
    l = np.full(n, 1 << 15, np.uint32)
    r = np.zeros(n, np.uint32)
    c[777] = l[777] = 0
    want = np.zeros(n, np.uint64)
    want[777] = 14772512
    for _ in range(20):
        got = gpu.count_tasks(16, c, l, r, per_task=True)
        assert np.array_equal(got["per_task"], want)


@pytest.mark.parametrize("N,k", [(14, 2), (16, 2)])
def test_dihedral_levels_keep_their_class(gpu, N, k):
    c, l, r, cls, _ = gpu.dihedral_expand(N, k)
    want = oracle.dihedral_count_tasks(N, k, c, l, r, cls)
    for _ in range(3):
        got = gpu.count_dihedral_tasks(N, k, c, l, r, cls, per_task=True)
        assert np.array_equal(got["per_task"], want)


def test_time_limit_still_stops(gpu):
    with pytest.raises(gpu.NQError) as e:
        gpu.count(19, 3, config=dict(time_limit_ms=3))
    assert e.value.status == gpu.NQ_ERR_TIMEOUT
    assert gpu.count(15, 2).total == 2279184


# 1024 threads and 14 slots fill the SM's shared memory, so the in-place step's
# extra slot does not fit; 13 leave room for one, 12 for the two that per-task
# counts take; 32 is the deepest stack.
@pytest.mark.parametrize("threads,levels", [(1024, 14), (1024, 13), (1024, 12), (448, 32), (416, 32), (32, 8)])
def test_stack_shapes_with_and_without_the_extra_slots(gpu, threads, levels):
    N, k = 13, 2
    c, l, r = oracle.expand(N, k)
    want = oracle.count_tasks(N, c, l, r)
    cfg = dict(block_threads=threads, stack_levels=levels)
    assert np.array_equal(gpu.count_tasks(N, c, l, r, per_task=True, config=cfg)["per_task"], want)
    res = gpu.count(N, k, config=cfg)
    assert res.total == 2 * int(want.sum()) and res.stats["stack_levels"] == levels
