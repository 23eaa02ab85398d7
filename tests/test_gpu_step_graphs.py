"""A step whose sizes repeat is replayed as a CUDA graph, small batches go through a pinned block, the head of a training step is one
kernel: the same numbers as launch by launch, and parity of the head at the edges of its register layouts."""
import numpy as np
import pytest

from goneuron_b200 import configs, descriptors as D
from tests.parity import TOL, assert_grads_close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    from goneuron_b200.sequential import Device
    d = Device(0)
    yield d
    d.close()


@pytest.mark.parametrize("name,kw,batch", [("mlp", {}, 24), ("cnn_bn", {}, 12), ("mlp_drop", {}, 24), ("lstm", dict(in_size=5, hidden=24, seq_len=7), 11),
                                           ("mlp", dict(in_size=3000, hidden=40), 64),                       # batch above the pinned block: copied in two parts
                                           ("transformer_small", dict(vocab=900, dim=128, seq_len=128, heads=2, ff_dim=512, n_blocks=2, causal=False), 16)])
def test_replayed_steps_equal_direct_ones(device, name, kw, batch):
    from goneuron_b200.sequential import Adam, Sequential
    layers, loss_kind, params, x, y, lr = configs.make_case(name, batch=batch, **kw)
    runs = []
    for direct in (1, 0):
        opt = Adam(lr)
        model = Sequential(layers, device).Compile(opt, loss_kind)
        model.SetParams(params)
        out = []
        for step in range(9):
            opt.LearningRate = lr * (1 + step)                            # a schedule: coefficients differ from replay to replay
            n = batch if step % 3 else batch // 2                         # two batch sizes in turn
            model.set_profiling(direct)                                   # (a profiled step is always issued launch by launch)
            out.append(model.TrainBatch(x[:n], y[:n]))
            if step % 4 == 1:
                out.append(model.PredictBatch(x[:n]))
            if step == 5:
                model.SetParams(params)
        model.set_profiling(0)
        runs.append((out, model.Params(), model.Gradients(), model.AdamState(), model.State()))
        model.Close()
    a, b = runs
    for u, v in zip(a[0], b[0]):
        assert np.array_equal(u, v)
    assert np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2]) and np.array_equal(a[4], b[4])
    assert all(np.array_equal(u, v) for u, v in zip(a[3], b[3]))


def test_graphs_follow_replaced_buffers(device):
    """Another model on the context grows the shared scratch, a larger batch replaces the model's own buffers: captured steps that
    refer to the old ones are not replayed."""
    from goneuron_b200.sequential import Adam, Sequential
    kw = dict(vocab=500, dim=128, seq_len=128, heads=2, ff_dim=512, n_blocks=2, causal=False)
    layers, loss_kind, params, x, y, lr = configs.make_case("transformer_small", batch=32, **kw)
    want = []
    for disturb in (False, True):
        model = Sequential(layers, device).Compile(Adam(lr), loss_kind)
        model.SetParams(params)
        for _ in range(3):
            model.TrainBatch(x[:8], y[:8])
        if disturb:
            l2, k2, p2, x2, y2, _ = configs.make_case("transformer_small", batch=48, **dict(kw, dim=256, heads=4))
            other = Sequential(l2, device).Compile(Adam(lr), k2)
            other.SetParams(p2); other.TrainBatch(x2, y2); other.Close()
        model.TrainBatch(x, y)
        for _ in range(3):
            model.TrainBatch(x[:8], y[:8])
        want.append(model.Params())
        model.Close()
    assert np.array_equal(*want)


@pytest.mark.parametrize("act,loss", [(D.LOGSOFTMAX, D.CROSS_ENTROPY), (D.SOFTMAX, D.CROSS_ENTROPY), (D.SOFTMAX, D.MSE)])
@pytest.mark.parametrize("n", [1, 2, 256, 257, 1025, 8191, 8193, 32768, 32769])
def test_head_parity(device, oracle, n, act, loss):
    from goneuron_b200.sequential import Adam, Sequential
    layers = [D.Dense(6, n, act)]
    rng = np.random.default_rng(n)
    params = (0.3 * rng.standard_normal(7 * n)).astype(np.float32)
    x = rng.standard_normal((3, 6)).astype(np.float32)
    y = np.zeros((3, n), np.float32); y[np.arange(3), rng.integers(0, n, 3)] = 1
    ref = oracle.OracleState(layers, loss, params, lr=1e-3)
    lit = oracle.OracleState(layers, loss, params, lr=1e-3)
    loss_ref = ref.train_batch(x, y, precision=64)
    lit.train_batch(x, y, precision=32)
    model = Sequential(layers, device).Compile(Adam(1e-3), loss)
    model.SetParams(params)
    got = model.TrainBatch(x, y)
    assert abs(got - loss_ref) <= TOL * max(1.0, abs(loss_ref))
    assert_grads_close(layers, model.Gradients(), ref.grads, floor=lit.grads)
    model.Close()


def test_a_failed_prediction_leaves_nothing_running(device):
    """Convolutions of some tens of milliseconds, then a layer that the library refuses: when the call returns its error, the stream is
    empty (the call's pinned block is the next call's), and the context goes on working."""
    import time
    from goneuron_b200 import _lib
    from goneuron_b200.sequential import Adam, Sequential
    hw = 1024
    layers = [D.Conv2D(1, 16, 7, 1, 3, D.RELU, hw, hw), D.Conv2D(16, 16, 7, 1, 3, D.RELU, hw, hw), D.MaxPool2D(16, 64, 64, 0, hw, hw),
              D.SequenceUnrollerLSTM(64, 512, 64, False), D.Dense(512, 2, D.LINEAR)]
    model = Sequential(layers, device).Compile(Adam(1e-3), D.MSE)
    x = np.random.default_rng(0).standard_normal((6, hw * hw)).astype(np.float32)
    times = []
    for _ in range(3):
        t0 = time.perf_counter()
        with pytest.raises(_lib.GoNeuronCudaError) as e:
            model.PredictBatch(x)
        t1 = time.perf_counter()
        device.synchronize()
        times.append((t1 - t0, time.perf_counter() - t1))
        assert e.value.code == -5 and "shared memory" in str(e.value)
    model.Close()
    call, wait = min(times)
    assert call + wait > 0.02 and wait < 0.1 * (call + wait), times
    l2, k2, p2, x2, y2, lr = configs.make_case("mlp", batch=8)
    other = Sequential(l2, device).Compile(Adam(lr), k2)
    other.SetParams(p2)
    assert np.isfinite(other.PredictBatch(x2)).all()
    other.Close()
