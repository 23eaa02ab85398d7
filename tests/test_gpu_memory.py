"""Device memory: what a failed allocation leaves behind."""
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
