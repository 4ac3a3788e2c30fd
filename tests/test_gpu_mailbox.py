"""When levels go through the mailbox between warps, and what happens there, on the GPU."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _device(gpu, N, tasks, per_task=True, config=None):
    import torch
    t = [torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda() for a in tasks]
    out = torch.zeros(2, dtype=torch.int64, device="cuda")
    per = torch.full((t[0].numel(),), -1, dtype=torch.int64, device="cuda") if per_task else None
    stream = torch.cuda.current_stream()

    def call():
        gpu.count_tasks_device(N, *t, out, per_task=per, config=config, stream=stream)

    call()
    torch.cuda.synchronize()
    assert int(out[1]) == 0
    return int(out[0]), per.cpu().numpy() if per_task else None, call


def _gpu_us(calls, reps=60):
    """Median GPU time of each call, taken in turn."""
    import torch
    times = [[] for _ in calls]
    for _ in range(reps):
        for call, ts in zip(calls, times):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            call()
            b.record()
            b.synchronize()
            ts.append(1e3 * a.elapsed_time(b))
    return [float(np.median(t)) for t in times]


# A list in device memory whose depth the caller does not state: the mailbox's rule
# must see the tasks' own depth (8 rows left), not that of an empty board, whose
# waits cost this list some 30 us a call.  Looking through the list costs 2-3 us.
def test_unstated_depth_costs_a_short_list_no_waits(gpu):
    N, k = 13, 5
    tasks = [a[:8000] for a in oracle.expand(N, k)]
    want = oracle.count_tasks(N, *tasks)
    stated = dict(stack_levels=gpu.stack_levels(N, k))
    for per_task in (False, True):
        got, per, plain = _device(gpu, N, tasks, per_task)
        assert got == int(want.sum()) and (not per_task or np.array_equal(per, want))
        _, _, told = _device(gpu, N, tasks, per_task, stated)
        a, b = _gpu_us((plain, told))
        assert a <= b + 15.0, (a, b)


# ... and must still see a deep task wherever it stands: 13 and 14 rows left, and one
# empty board among boards that are full or have columns off the board.
@pytest.mark.parametrize("N,k", [(13, 1), (15, 1), (15, 2)])
def test_unstated_depth_of_deep_lists(gpu, N, k):
    tasks = oracle.expand(N, k)
    want = oracle.count_tasks(N, *tasks)
    got, per, _ = _device(gpu, N, tasks)
    assert got == int(want.sum()) and np.array_equal(per, want)


@pytest.mark.parametrize("n,at", [(1, 0), (1023, 1022), (1025, 1024), (20000, 777), (400000, 399999)])
def test_unstated_depth_of_one_deep_task(gpu, n, at):
    c = np.full(n, (1 << 16) - 1, np.uint32)
    c[::3] = 1 << 20
    l, r = np.full(n, 1 << 15, np.uint32), np.zeros(n, np.uint32)
    c[at] = l[at] = 0
    got, per, call = _device(gpu, 16, (c, l, r))
    full = (c == (1 << 16) - 1).astype(np.int64)  # a finished board is one completion
    full[at] = 14772512
    assert got == int(full.sum()) and np.array_equal(per, full)
    # without the mailbox a single board of 1.3e9 nodes keeps a few warps busy for far longer
    assert _gpu_us((call,), 5)[0] < 20e3


def _count(gpu, N, tasks, config, nodes=False):
    """nq_count_tasks with per-task outputs, and the mailbox's tickets and posts."""
    c, l, r = tasks
    per, nd = (np.full(c.size, 9, np.uint64) for _ in range(2))
    total, st = ctypes.c_uint64(0), gpu.Stats()
    rc = gpu.lib.nq_count_tasks(N, *(gpu._p(a, gpu._u32p) for a in (c, l, r)), c.size, gpu._p(per, gpu._u64p),
                                gpu._p(nd, gpu._u64p) if nodes else None, ctypes.byref(total), gpu._cfg(config),
                                ctypes.byref(st))
    assert rc == 0, gpu.last_error()
    assert total.value == int(per.sum())
    return per, nd, st.reserved[0], st.reserved[1]


# reserved[0] = 1 + the wait limit in us: no patience at all, and waits that end while
# levels are being offered; both leave tickets that posters find given up.
@pytest.mark.parametrize("limit_us", [0, 5, 50])
@pytest.mark.parametrize("N,k", [(15, 1), (15, 2)])
def test_waits_for_mail_that_run_out(gpu, N, k, limit_us):
    tasks = oracle.expand(N, k)
    want, want_nodes = oracle.count_tasks(N, *tasks, nodes=True)
    tickets = posts = 0
    for cfg in (dict(), dict(block_threads=32, blocks_per_sm=1), dict(block_threads=256, layout=1)):
        cfg["reserved"] = (1 + limit_us, 0)
        for nodes in (False, True):
            per, nd, t, p = _count(gpu, N, tasks, cfg, nodes)
            assert np.array_equal(per, want) and (not nodes or np.array_equal(nd, want_nodes)), cfg
            tickets, posts = tickets + t, posts + p
    assert tickets > 0 and posts > 0
    # the scratch is as a launch with the usual patience needs it
    assert np.array_equal(_count(gpu, N, tasks, None)[0], want)


def test_dihedral_and_batch_waits_that_run_out(gpu):
    c, l, r, cls, _ = gpu.dihedral_expand(16, 2)
    want = oracle.dihedral_count_tasks(16, 2, c, l, r, cls)
    boards = [(15, 0, 0, 0), (16, 1, 2, 0), (14, 0, 0, 0), (13, 2, 4, 1)]
    counts = [oracle.count_task(*b) for b in boards]
    for reserved in ((1, 0), (6, 0), (51, 0), (0, 0)):
        got = gpu.count_dihedral_tasks(16, 2, c, l, r, cls, per_task=True, config=dict(reserved=reserved))
        assert np.array_equal(got["per_task"], want)
        assert gpu.count_batch(boards, split_rows=1, config=dict(reserved=reserved)).tolist() == counts


# One warp per SM and the smallest ring above twice their number: a heavy board draws
# more tickets than the ring has slots, so slots go into later uses.
@pytest.mark.parametrize("limit_us", [None, 200])
def test_ring_slots_are_used_again(gpu, limit_us):
    n = 3000
    c, l, r = np.full(n, (1 << 17) - 1, np.uint32), np.full(n, 1 << 16, np.uint32), np.zeros(n, np.uint32)
    c[1234] = l[1234] = 0
    want = np.ones(n, np.uint64)
    want[1234] = 95815104
    cfg = dict(block_threads=32, blocks_per_sm=1, reserved=(0 if limit_us is None else 1 + limit_us, 512))
    for _ in range(3):
        per, _, tickets, posts = _count(gpu, 17, (c, l, r), cfg)
        assert np.array_equal(per, want)
        if limit_us is None:
            assert tickets > 512 and posts > 512, (tickets, posts)
    assert np.array_equal(_count(gpu, 17, (c, l, r), None)[0], want)


# The stack a caller asks for does not decide about the mailbox: eight rows are left.
def test_a_deeper_stack_does_not_switch_the_mailbox_on(gpu):
    tasks = [a[:8000] for a in oracle.expand(13, 5)]
    want = oracle.count_tasks(13, *tasks)
    for cfg in (None, dict(stack_levels=20), dict(stack_levels=32)):
        per, _, tickets, posts = _count(gpu, 13, tasks, cfg)
        assert np.array_equal(per, want) and tickets == posts == 0
