"""The cost model at its limits, on the GPU: waits for the tensor cores that expire, infinite and huge weights,
the order of the gradient's sums."""
import ctypes

import numpy as np
import pytest

import oracle
from oracle import mlp_ref

pytestmark = pytest.mark.gpu
POLLS = 1 << 22  # the default limit


def _params(seed):
    p = np.random.default_rng(seed).uniform(-0.12, 0.12, mlp_ref.NPARAMS).astype(np.float32)
    p[mlp_ref.OFF_B3] = 12.0
    return p


def _schedule(learned, m, N, tasks, last=None):
    import torch
    t = [torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda() for a in tasks]
    order = torch.full((t[0].numel(),), -1, dtype=torch.int32, device="cuda")
    d_last = None if last is None else torch.tensor(last, dtype=torch.int32, device="cuda")
    rc = learned.lib.nq_schedule_device_last(m._m, N, *(a.data_ptr() for a in t), order.numel(),
                                             d_last.data_ptr() if last else None, len(last or ()), order.data_ptr(),
                                             None, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    return order.cpu().numpy()


# one task; a ragged tile; more tiles than the 148 x 4 groups, so that a group leaves several unfinished
@pytest.mark.parametrize("n", [1, 300, 75_777, 200_001])
def test_expired_wait_leaves_a_permutation_and_is_reported(gpu, n):
    from n_queens_b200 import learned
    N = 17
    tasks = [a[:n] for a in oracle.expand(N, 6)]
    m = learned.CostModel(seed=3)
    m.set_params(_params(3))
    pred, order = m.predict(N, *tasks), _schedule(learned, m, N, tasks)
    learned.lib.nq_mlp_set_wait_limit(m._m, 0)
    assert np.array_equal(_schedule(learned, m, N, tasks), np.arange(n))
    last = [0, n // 2] if n > 2 else []
    want = np.concatenate([np.setdiff1d(np.arange(n), last), np.array(last, np.int64)])
    assert np.array_equal(_schedule(learned, m, N, tasks, last), want)
    for f in (m.predict, m.predict_tensor):
        with pytest.raises(gpu.NQError) as e:
            f(N, *tasks)
        assert e.value.status == gpu.NQ_ERR_TIMEOUT
    learned.lib.nq_mlp_set_wait_limit(m._m, POLLS)
    assert np.array_equal(m.predict(N, *tasks), pred) and np.array_equal(_schedule(learned, m, N, tasks), order)
    m.close()


def test_learned_count_reports_an_expired_wait_with_the_right_total(gpu):
    from n_queens_b200 import learned
    m = learned.CostModel(seed=3)
    for polls, status in ((0, gpu.NQ_ERR_TIMEOUT), (POLLS, gpu.NQ_OK), (0, gpu.NQ_ERR_TIMEOUT)):
        learned.lib.nq_mlp_set_wait_limit(m._m, polls)
        total = ctypes.c_uint64(0)
        assert learned.lib.nq_count_learned(14, 4, m._m, None, ctypes.byref(total), None) == status
        assert total.value == 365596
    m.close()


def _forward_over_set_bits(p, X):
    """Float64 forward that adds only the W1 columns of the set bits, ReLU of NaN = 0 (CUDA's fmaxf)."""
    W1, b1, W2, b2, W3, b3 = mlp_ref.unpack(p)
    with np.errstate(all="ignore"):
        h1 = np.stack([np.fmax(b1 + W1[:, x > 0].sum(1), 0) for x in X])
        h2 = np.fmax((h1[:, None, :] * W2[None]).sum(2) + b2, 0)
        return (h2 * W3).sum(1) + b3


# Column 20 is off the N=14 board (no input bit), column 3 is on it.  2^32 is where
# the general forward takes over.  FP32 sums of 96 and 128 terms: 1e-5 of the largest output.
@pytest.mark.parametrize("where,value", [
    (5 * 96 + 20, np.inf), (5 * 96 + 20, np.nan), (5 * 96 + 20, 3e38), (5 * 96 + 3, np.inf), (5 * 96 + 3, -np.inf),
    (5 * 96 + 3, np.nan), (5 * 96 + 3, 1e37), (5 * 96 + 3, 2.0**32), (5 * 96 + 3, 2.0**31), (mlp_ref.OFF_B1 + 5, 3.395e38),
    (mlp_ref.OFF_B1 + 5, np.inf), (mlp_ref.OFF_W2 + 7, np.inf), (mlp_ref.OFF_W2 + 7, -np.inf), (mlp_ref.OFF_W2 + 7, 1e30),
    (mlp_ref.OFF_B2 + 7, np.nan), (mlp_ref.OFF_B2 + 7, 1e33), (mlp_ref.OFF_W3 + 7, np.inf), (mlp_ref.OFF_B3, np.inf)])
@pytest.mark.parametrize("n", [1, 300])
def test_predictions_with_infinite_and_huge_weights(gpu, where, value, n):
    from n_queens_b200 import learned
    p = _params(1)
    p[where] = value
    c, l, r = (a[:n] for a in oracle.expand(14, 5))
    m = learned.CostModel(seed=3)
    m.set_params(p)
    got, want = m.predict(14, c, l, r), _forward_over_set_bits(p, mlp_ref.features(14, c, l, r))
    finite = np.isfinite(want)
    assert np.array_equal(got[~finite], want[~finite].astype(np.float32), equal_nan=True)
    if finite.any():
        assert np.abs(got[finite] - want[finite]).max() <= 1e-5 * np.abs(want[finite]).max()
    m.close()


def test_weight_gradient_sums_tile_by_tile(gpu):
    # Weights and labels on binary grids, so that the forward pass and every factor of
    # dW2 are exact in FP32 and only the order of its sums shows; labels around the
    # prediction, so that the terms cancel.  131072 tasks are 28 tiles for each of 148
    # CTAs: a CPU emulation of both orders gives an error of 2.2e-7 with a sum per tile
    # and 5.7e-7 with one running sum over a CTA's tiles.
    from n_queens_b200 import learned
    n, rng = 1 << 17, np.random.default_rng(1)
    p = np.zeros(mlp_ref.NPARAMS, np.float32)
    p[:mlp_ref.OFF_W3] = rng.integers(-8, 9, mlp_ref.OFF_W3) / 64
    p[mlp_ref.OFF_B1:mlp_ref.OFF_W2] = rng.integers(-512, 513, mlp_ref.H1) / 4096
    p[mlp_ref.OFF_W3:mlp_ref.OFF_B3] = rng.choice([-0.125, 0.125], mlp_ref.H2)
    tasks = [a[:n] for a in oracle.expand(17, 6)]
    X = mlp_ref.features(17, *tasks)
    out = mlp_ref.forward(p, X)[0]
    y = ((np.round(out * 2**20) + rng.integers(-2**22, 2**22, n)) / 2**20).astype(np.float32)
    want = mlp_ref.loss_and_grad(p, X, y)[1]
    m = learned.CostModel(seed=3)
    m.set_params(p)
    got = m.grad(np.full(n, 17, np.uint8), *tasks, y)[0]
    m.close()
    w2 = slice(mlp_ref.OFF_W2, mlp_ref.OFF_B2)
    assert np.linalg.norm(got[w2] - want[w2]) <= 3.5e-7 * np.linalg.norm(want[w2])


def _gradient_over_set_bits(p, X, y):
    """Float64 gradient by the sums that the model states: layer 1 and dW1 over set bits only."""
    W1, b1, W2, b2, W3, b3 = mlp_ref.unpack(p)
    with np.errstate(all="ignore"):
        h1 = np.stack([np.fmax(b1 + W1[:, x > 0].sum(1), 0) for x in X])
        h2 = np.fmax((h1[:, None, :] * W2[None]).sum(2) + b2, 0)
        e = (h2 * W3).sum(1) + b3 - y
        d = 2.0 / len(y) * e
        dh2 = np.where(h2 > 0, d[:, None] * W3, 0.0)
        dh1 = np.where(h1 > 0, (dh2[:, :, None] * W2[None]).sum(1), 0.0)
        dw1 = np.stack([dh1[X[:, f] > 0].sum(0) for f in range(mlp_ref.IN)], 1)
        parts = (dw1, dh1.sum(0), (dh2[:, :, None] * h1[:, None, :]).sum(0), dh2.sum(0), (d[:, None] * h2).sum(0),
                 [d.sum()])
        return (e * e).mean(), np.concatenate([np.asarray(q).ravel() for q in parts])


# One task (31 rows of the tile unused), one more than a tile, ragged tiles.  where < 0: the label of task 0.
@pytest.mark.parametrize("n", [1, 33, 300])
@pytest.mark.parametrize("where,value", [
    (-1, np.nan), (-1, np.inf), (5 * 96 + 20, np.inf), (5 * 96 + 3, np.inf), (5 * 96 + 3, np.nan),
    (mlp_ref.OFF_B1 + 5, np.inf), (mlp_ref.OFF_W2 + 7, np.inf), (mlp_ref.OFF_B2 + 7, np.inf),
    (mlp_ref.OFF_W3 + 7, np.inf), (mlp_ref.OFF_W3 + 7, np.nan), (mlp_ref.OFF_B3, np.inf)])
def test_gradient_with_infinities(gpu, where, value, n):
    from n_queens_b200 import learned
    p, y = _params(1), np.random.default_rng(2).normal(12, 1.5, n).astype(np.float32)
    if where < 0:
        y[0] = value
    else:
        p[where] = value
    tasks = [a[:n] for a in oracle.expand(14, 5)]
    m = learned.CostModel(seed=3)
    m.set_params(p)
    got, loss = m.grad(np.full(n, 14, np.uint8), *tasks, y)
    m.close()
    want_loss, want = _gradient_over_set_bits(p, mlp_ref.features(14, *tasks), y.astype(np.float64))
    finite = np.isfinite(want)
    assert np.array_equal(got[~finite], want[~finite].astype(np.float32), equal_nan=True)
    # FP32 sums of up to 300 terms, after layers of 96 and 128
    assert np.abs(got[finite] - want[finite]).max() <= 1e-5 * np.abs(want[finite]).max()
    assert np.isfinite(loss) == np.isfinite(want_loss)


def test_error_words_of_many_models(gpu):
    # more models at once than one page of error words holds; a failure shows in its own model only
    from n_queens_b200 import learned
    tasks = [a[:200] for a in oracle.expand(14, 5)]
    models = [learned.CostModel(seed=k) for k in range(70)]
    for k in (0, 63, 64, 69):
        learned.lib.nq_mlp_set_wait_limit(models[k]._m, 0)
    for k, m in enumerate(models):
        if k in (0, 63, 64, 69):
            with pytest.raises(gpu.NQError):
                m.predict(14, *tasks)
        else:
            m.predict(14, *tasks)
    for m in models:
        m.close()
    m = learned.CostModel(seed=0)  # takes a slot that a model before it has used
    m.predict(14, *tasks)
    m.close()
