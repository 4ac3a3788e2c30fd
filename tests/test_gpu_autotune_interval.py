"""The autotuner's sweep measures the launch that a plan takes by itself, on the GPU."""
import pytest

from n_queens_b200 import workloads

pytestmark = pytest.mark.gpu


def test_sweep_runs_the_interval_of_a_default_plan(gpu):
    # Fewer than four subtasks per lane at every split depth: such plans visit the queue every 256 steps.
    inst = workloads.random_boards(32, 4, 8, 9, 0, 3)
    best, table = gpu.autotune_batch(inst, repeats=1)
    assert [e["inner_steps"] for e in table] == [256] * 40 + [1024, 4096]
    assert best in table


def test_sweep_keeps_a_stated_interval(gpu):
    inst = workloads.random_boards(32, 4, 8, 9, 0, 3)
    for inner, rest in ((62, [256, 4096]), (1024, [256, 4096]), (256, [4096])):
        _, table = gpu.autotune_batch(inst, repeats=1, config=dict(inner_steps=inner))
        assert [e["inner_steps"] for e in table] == [(inner + 3) // 4 * 4] * 40 + rest
