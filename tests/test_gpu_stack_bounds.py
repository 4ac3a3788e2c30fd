"""Stated stack depths at their bounds: what nq_stack_levels states is taken, one slot less is refused."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,k", [(12, 4), (13, 2)])
@pytest.mark.parametrize("outputs", ["sum", "per_task", "nodes"])
def test_device_entry_refuses_one_slot_less(gpu, N, k, outputs):
    import torch
    tasks = oracle.expand(N, k)
    want, nodes = oracle.count_tasks(N, *tasks, nodes=True)
    t = [torch.from_numpy(a.view(np.int32)).cuda() for a in tasks]
    levels = gpu.stack_levels(N, k, outputs == "nodes")
    for less in (0, 1):
        out = torch.zeros(2, dtype=torch.int64, device="cuda")
        per, nd = (torch.zeros(want.size, dtype=torch.int64, device="cuda") for _ in range(2))
        gpu.count_tasks_device(N, *t, out, per_task=None if outputs == "sum" else per,
                               nodes=nd if outputs == "nodes" else None, config=dict(stack_levels=levels - less))
        torch.cuda.synchronize()
        assert int(out[1]) == less  # status bit 1: a task needed more stack levels than the launch had
        if not less:
            assert int(out[0]) == int(want.sum())
            assert outputs == "sum" or np.array_equal(per.cpu().numpy(), want.astype(np.int64))
            assert outputs != "nodes" or np.array_equal(nd.cpu().numpy(), nodes.astype(np.int64))


@pytest.mark.parametrize("kind", ["count", "nodes", "dihedral"])
def test_host_entries_refuse_one_slot_less(gpu, kind):
    N, k = 12, 4
    levels = gpu.stack_levels(N, k, kind != "count")
    call = {"count": lambda **c: gpu.count(N, k, **c).total, "nodes": lambda **c: gpu.count(N, k, nodes=True, **c).total,
            "dihedral": lambda **c: gpu.count_dihedral(N, k, **c).total}[kind]
    assert call(config=dict(stack_levels=levels)) == 14200
    with pytest.raises(gpu.NQError) as e:
        call(config=dict(stack_levels=levels - 1))
    assert e.value.status == gpu.NQ_ERR_DEPTH
