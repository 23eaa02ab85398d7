"""Device memory: what a failed allocation leaves behind, and what becomes of the buffers of closed models."""
import numpy as np
import pytest

from goneuron_b200 import configs, descriptors as D

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    from goneuron_b200.sequential import Device
    d = Device(0)
    yield d
    d.close()


@pytest.mark.parametrize("name,kw,huge", [("transformer_small", dict(vocab=300, dim=64, seq_len=512, heads=2, ff_dim=96, n_blocks=2), 1 << 20), ("mlp", {}, 1 << 27)])
@pytest.mark.parametrize("before", [True, False])
def test_out_of_memory_is_an_error_and_nothing_else(device, name, kw, huge, before):
    """A batch whose activations exceed the device (400 GB and more) is refused with GN_ERR_OOM, which loses the old buffers; the calls after it
    work as on a fresh model.  (Its device pointers are never read.)"""
    from goneuron_b200 import _lib
    from goneuron_b200.sequential import Adam, Sequential
    layers, loss_kind, params, x, y, lr = configs.make_case(name, batch=4, **kw)
    got = []
    for fail in (False, True):
        model = Sequential(layers, device).Compile(Adam(lr), loss_kind)
        model.SetParams(params)
        out = [model.PredictBatch(x), model.TrainBatch(x, y), model.TrainBatch(x, y)] if before else []
        if fail:
            xd, yd = device.alloc(x), device.alloc(y)
            with pytest.raises(_lib.GoNeuronCudaError) as e:
                model.TrainBatchDevice(xd, yd, huge)
            assert e.value.code == -7, e.value
            device.free(xd); device.free(yd)
        out += [model.PredictBatch(x[:2]), model.TrainBatch(x[:3], y[:3]), model.TrainBatch(x, y), model.PredictBatch(x), model.Params()]
        got.append(out)
        model.Close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


def _model(device, batch, **kw):
    from goneuron_b200.sequential import Adam, Sequential
    layers, loss_kind, params, x, y, lr = configs.make_case("transformer_small", batch=batch, **dict(dict(vocab=500, dim=256, seq_len=256, heads=8, ff_dim=1024, n_blocks=4, causal=False), **kw))
    model = Sequential(layers, device).Compile(Adam(lr), loss_kind)
    model.SetParams(params)
    out = [model.TrainBatch(x, y), model.PredictBatch(x)]
    return model, out + [model.TrainBatch(x, y), model.Params()]


def test_memory_of_closed_models(device):
    """The driver gets everything back when the last model closes; while one lives, what a closed one held serves the next (same results in
    buffers that are not fresh)."""
    small, _ = _model(device, 2)
    small.Close()                                             # (the context's own scratch has its size for batches of two from here on)
    before = _free()
    a, want = _model(device, 2)
    b, _ = _model(device, 160)                                # about 3 GB
    full = _free()
    assert before - full > 2 << 30
    b.Close()
    for _ in range(2):
        c, got = _model(device, 2)
        c.Close()
        assert all(np.array_equal(u, v) for u, v in zip(got, want))
    b, _ = _model(device, 160)
    assert abs(_free() - full) < 64 << 20                     # nothing was asked of the driver twice
    b.Close(); a.Close()
    assert before - _free() < 1 << 30                         # what is left: the context's scratch for the large batch


def test_kept_memory_serves_other_sizes_when_the_device_is_full(device):
    """With no memory left at the driver a model of another size gets what closed ones have left behind."""
    import torch
    a, _ = _model(device, 2)
    b, _ = _model(device, 160)
    b.Close()                                                 # some 3 GB, kept because `a` lives
    held = torch.empty(_free() - (600 << 20), dtype=torch.uint8, device="cuda")
    try:
        c, got = _model(device, 100, seq_len=224)             # other sizes, 1.5 GB
        c.Close()
    finally:
        del held
        torch.cuda.empty_cache()
    c, want = _model(device, 100, seq_len=224)
    c.Close(); a.Close()
    assert all(np.array_equal(u, v) for u, v in zip(got, want))
