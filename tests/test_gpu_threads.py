"""Several threads on one GPU: steps that are recorded and replayed in one of them, everything else that a program may do at the same time
in the others."""
import threading

import numpy as np
import pytest

from goneuron_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    from goneuron_b200.sequential import Device
    d = Device(0)
    yield d
    d.close()


CASES = [("mlp", {}, 24), ("lstm", dict(in_size=5, hidden=24, seq_len=7), 11),
         ("transformer_small", dict(vocab=900, dim=128, seq_len=128, heads=2, ff_dim=512, n_blocks=2, causal=False), 8)]


def _train(device, rounds):
    """New models again and again, so that steps are recorded all the time."""
    from goneuron_b200.sequential import Adam, Sequential
    out = []
    for _ in range(rounds):
        for name, kw, batch in CASES:
            layers, loss_kind, params, x, y, lr = configs.make_case(name, batch=batch, **kw)
            model = Sequential(layers, device).Compile(Adam(lr), loss_kind)
            model.SetParams(params)
            for n in (batch, batch, batch // 2, batch // 2, batch, batch // 2):
                out.append(model.TrainBatch(x[:n], y[:n]))
                out.append(model.PredictBatch(x[:n]).copy())
            out.append(model.Params())
            model.Close()
    return out


def _disturb(device, stop, own_device):
    """What another thread may do: its own model's state, device memory, waiting for the stream and for the whole device, models that
    come and go."""
    import torch
    from goneuron_b200.sequential import Adam, Device, Sequential
    layers, loss_kind, params, x, y, lr = configs.make_case("mlp", batch=8)
    dev = Device(0) if own_device else device
    k = 0
    while not stop.is_set():
        model = Sequential(layers, dev).Compile(Adam(lr), loss_kind)
        for _ in range(20):
            k += 1
            p = params + np.float32(k)
            model.SetParams(p)
            model.SetAdamState(p, np.abs(p), k)
            torch.cuda.synchronize()
            assert np.array_equal(model.Params(), p)
            assert np.array_equal(model.AdamState()[0], p) and not model.Gradients().any()
            d = dev.alloc(x)
            dev.synchronize()
            dev.free(d)
        model.Close()
    if own_device:
        dev.close()


@pytest.mark.parametrize("own_device", [False, True])
def test_steps_are_recorded_while_other_threads_work(device, own_device):
    want = _train(device, 1)
    stop, errors = threading.Event(), []

    def guarded():
        try:
            _disturb(device, stop, own_device)
        except BaseException as e:                           # noqa: BLE001 (handed to the test's thread)
            errors.append(e)
    threads = [threading.Thread(target=guarded) for _ in range(2)]
    for t in threads:
        t.start()
    try:
        got = _train(device, 6)
    finally:
        stop.set()
        for t in threads:
            t.join(60)
    assert not errors, errors[0]
    for k, v in enumerate(got):
        assert np.array_equal(v, want[k % len(want)]), k


def test_two_threads_train_on_one_device(device):
    want = _train(device, 1)
    got = [None, None]

    def work(i):
        got[i] = _train(device, 3)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    for g in got:
        assert g is not None
        for k, v in enumerate(g):
            assert np.array_equal(v, want[k % len(want)]), k
