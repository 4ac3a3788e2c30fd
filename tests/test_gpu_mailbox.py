"""When levels go through the mailbox between warps, and what happens there, on the GPU."""
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
