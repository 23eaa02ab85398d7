"""The register-tiled convolution kernels (engine 0 of gn_op_conv2d) where their tiling can go wrong: widths that are no multiple of four,
channel counts around the groups of eight, images taller than a band, several source-channel chunks, one image and many, and
the pooling gradient's two forms -- against float64 numpy."""
import ctypes as C

import numpy as np
import pytest

from goneuron_b200 import configs, descriptors as D
from tests.parity import TOL, assert_grads_close, norm_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    from goneuron_b200.sequential import Device
    d = Device(0)
    yield d
    d.close()


def _f(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


@pytest.mark.parametrize("B,inC,outC,k,p,H,W,act", [
    (1, 1, 1, 1, 0, 1, 1, D.LINEAR), (2, 3, 8, 1, 0, 5, 7, D.RELU), (3, 9, 17, 3, 1, 7, 6, D.RELU), (2, 5, 7, 3, 0, 9, 10, D.TANH), (1, 33, 40, 3, 2, 12, 13, D.RELU),
    (200, 1, 24, 3, 1, 28, 28, D.RELU), (2, 70, 65, 3, 1, 8, 8, D.LINEAR), (3, 4, 6, 5, 2, 31, 33, D.SIGMOID), (2, 40, 9, 5, 4, 6, 5, D.RELU), (1, 2, 3, 3, 1, 300, 301, D.RELU),
    (2, 3, 100, 3, 1, 40, 40, D.RELU), (4, 16, 4, 3, 1, 2, 3, D.LINEAR),
    # windows that keep an image of whole 16-byte pieces: widths of 4 to 508, odd heights, channels dealt out to one, two and four groups, more than are staged at once
    (3, 5, 6, 3, 1, 3, 4, D.TANH), (2, 9, 18, 3, 1, 7, 8, D.RELU), (2, 17, 33, 5, 2, 9, 16, D.RELU), (1, 8, 20, 3, 1, 4, 508, D.LINEAR), (2, 130, 19, 3, 1, 11, 20, D.TANH), (5, 20, 12, 1, 0, 5, 12, D.RELU),
    # other activations: a row per thread (windows of every size, both ways of staging, narrow images, bands of few rows), and two rows (many threads)
    (4, 3, 9, 5, 2, 7, 8, D.TANH), (3, 4, 6, 3, 1, 9, 16, D.SIGMOID), (100, 1, 12, 3, 1, 28, 28, D.TANH), (3, 6, 7, 1, 0, 5, 12, D.SIGMOID), (2, 3, 5, 1, 0, 4, 6, D.TANH), (2, 3, 9, 5, 0, 14, 15, D.TANH),
    (70, 9, 33, 3, 1, 17, 32, D.TANH), (90, 8, 30, 3, 0, 19, 33, D.SIGMOID),
    (200, 16, 32, 1, 0, 16, 16, D.RELU), (200, 16, 16, 5, 2, 12, 12, D.RELU), (60, 24, 24, 1, 0, 30, 30, D.TANH),      # input gradients of many threads: two rows, and 1 x 1 windows in one
    (2, 3, 4, 3, 1, 5, 513, D.RELU), (1, 2, 5, 5, 2, 7, 520, D.TANH), (1, 2, 3, 3, 3, 6, 9, D.RELU), (1, 2, 3, 1, 0, 3, 600, D.RELU)])      # the plain kernels' side of the limits
def test_conv_direct(device, B, inC, outC, k, p, H, W, act):
    from goneuron_b200 import _lib
    oH, oW = H + 2 * p - k + 1, W + 2 * p - k + 1
    rng = np.random.default_rng(B * 1000 + inC * 100 + outC * 10 + k)
    x, w = rng.standard_normal((B, inC, H, W)).astype(np.float32), (rng.standard_normal((outC, inC, k, k)) / np.sqrt(inC * k * k)).astype(np.float32)
    bias, dy = rng.standard_normal(outC).astype(np.float32), rng.standard_normal((B, outC, oH, oW)).astype(np.float32)
    y, dx, dw, db = np.empty((B, outC, oH, oW), np.float32), np.empty_like(x), np.empty_like(w), np.empty_like(bias)
    _lib.check(_lib.load().gn_op_conv2d(device.handle, 0, B, inC, outC, k, 1, p, H, W, act, _f(x), _f(w), _f(bias), _f(dy), _f(y), _f(dx), _f(dw), _f(db)))
    xp = np.pad(x.astype(np.float64), ((0, 0), (0, 0), (p, p), (p, p)))
    z = np.zeros((B, outC, oH, oW)) + bias.astype(np.float64)[None, :, None, None]
    for i in range(k):
        for j in range(k):
            z += np.einsum("bchw,oc->bohw", xp[:, :, i:i + oH, j:j + oW], w[:, :, i, j].astype(np.float64), optimize=True)
    a = {D.LINEAR: z, D.RELU: np.maximum(z, 0), D.TANH: np.tanh(z), D.SIGMOID: 1 / (1 + np.exp(-z))}[act]
    der = {D.LINEAR: np.ones_like(z), D.RELU: y > 0, D.TANH: 1 - a * a, D.SIGMOID: a * (1 - a)}[act]      # (ReLU: the pattern of the result itself)
    assert norm_err(y, a) <= 1e-5
    dz = dy * der
    dxp, dwr = np.zeros_like(xp), np.zeros(w.shape)
    for i in range(k):
        for j in range(k):
            dxp[:, :, i:i + oH, j:j + oW] += np.einsum("bohw,oc->bchw", dz, w[:, :, i, j].astype(np.float64), optimize=True)
            dwr[:, :, i, j] = np.einsum("bohw,bchw->oc", dz, xp[:, :, i:i + oH, j:j + oW], optimize=True)
    dxr = dxp[:, :, p:p + H, p:p + W]
    assert norm_err(dx, dxr) <= 1e-5 and norm_err(dw, dwr) <= 1e-5 and norm_err(db, dz.sum((0, 2, 3))) <= 1e-5


@pytest.mark.parametrize("k,s,p,hw", [(2, 2, 0, 9), (2, 3, 1, 10), (3, 3, 1, 11), (3, 2, 1, 9), (1, 2, 0, 7)])
def test_maxpool_gradient(device, oracle, k, s, p, hw):
    from goneuron_b200.sequential import Adam, Sequential
    o = (hw + 2 * p - k) // s + 1
    layers = [D.Conv2D(2, 3, 3, 1, 1, D.TANH, hw, hw), D.MaxPool2D(3, k, s, p, hw, hw), D.Flatten(), D.Dense(3 * o * o, 4, D.SOFTMAX)]
    rng = np.random.Generator(np.random.PCG64(k * 10 + s))
    params = configs.init_params(layers, rng)
    x, y = configs.make_inputs("cnn", layers, 5, rng)
    ref = oracle.OracleState(layers, D.CROSS_ENTROPY, params, lr=1e-3)
    ref.train_batch(x, y, precision=64)
    model = Sequential(layers, device).Compile(Adam(1e-3), D.CROSS_ENTROPY)
    model.SetParams(params)
    model.TrainBatch(x, y)
    assert_grads_close(layers, model.Gradients(), ref.grads)
    model.Close()


def test_maxpool_of_a_large_plane(device):
    """More than 65 535 x 256 pixels: a block takes several pieces of the plane, in all three kernels."""
    from goneuron_b200.sequential import Adam, Sequential
    hw = 8194                                                 # halves to 4097 x 4097 = 16.8 M pixels, then to 17 x 17
    layers = [D.MaxPool2D(1, 2, 2, 0, hw, hw), D.MaxPool2D(1, 241, 241, 0, hw // 2, hw // 2), D.Flatten(), D.Dense(289, 2, D.LINEAR)]
    rng = np.random.default_rng(2)
    params = rng.standard_normal(289 * 2 + 2).astype(np.float32)
    x, y = rng.standard_normal((1, hw * hw), dtype=np.float32), np.array([[1.0, -2.0]], np.float32)
    model = Sequential(layers, device).Compile(Adam(1e-3), D.MSE)
    model.SetParams(params)
    p = x.reshape(17, 482, 17, 482).max((1, 3)).reshape(1, 289).astype(np.float64)
    out = p @ params[:578].reshape(2, 289).T.astype(np.float64) + params[578:]
    assert norm_err(model.PredictBatch(x), out) <= 1e-5
    model.TrainBatch(x, y)                                    # (runs the gradients of both layers)
    g = model.Gradients()
    assert norm_err(g[:578].reshape(2, 289), (out - y).T @ p) <= 1e-5
    model.Close()


def test_batchnorm_running_statistics_of_a_long_batch(device, oracle):
    """More samples than a block stages at a time, more channels than a block has lanes."""
    from goneuron_b200.sequential import Adam, Sequential
    layers = [D.Conv2D(1, 40, 1, 1, 0, D.LINEAR, 4, 4), D.BatchNorm2D(40, 4, 4), D.Flatten(), D.Dense(640, 3, D.SOFTMAX)]
    rng = np.random.Generator(np.random.PCG64(8))
    params = configs.init_params(layers, rng)
    x, y = configs.make_inputs("cnn_bn", layers, 300, rng)
    ref = oracle.OracleState(layers, D.CROSS_ENTROPY, params, lr=1e-3)
    ref.train_batch(x, y, precision=64)
    model = Sequential(layers, device).Compile(Adam(1e-3), D.CROSS_ENTROPY)
    model.SetParams(params)
    model.TrainBatch(x, y)
    assert norm_err(model.State(), ref.state) <= TOL
    model.Close()


ANY_POINTER = {
    "conv 5x5": [D.Conv2D(3, 6, 5, 1, 0, D.RELU, 12, 16), D.Flatten(), D.Dense(6 * 8 * 12, 4, D.SOFTMAX)],
    "conv 1x1": [D.Conv2D(4, 9, 1, 1, 0, D.TANH, 8, 8), D.Flatten(), D.Dense(9 * 64, 4, D.SOFTMAX)],
    "conv 3x3": [D.Conv2D(2, 5, 3, 1, 1, D.RELU, 8, 8), D.Flatten(), D.Dense(5 * 64, 4, D.SOFTMAX)],
    "pool": [D.MaxPool2D(3, 2, 2, 0, 8, 8), D.Flatten(), D.Dense(48, 4, D.SOFTMAX)],
    "batch norm": [D.BatchNorm2D(3, 8, 8), D.Flatten(), D.Dense(192, 4, D.SOFTMAX)],
    "dense": [D.Dense(64, 32, D.RELU), D.Dense(32, 4, D.SOFTMAX)],
    "wide dense": [D.Dense(512, 640, D.RELU), D.Dense(640, 4, D.SOFTMAX)],
    "lstm": [D.SequenceUnrollerLSTM(8, 16, 6, False), D.Dense(16, 4, D.SOFTMAX)],
    "gru": [D.SequenceUnrollerGRU(8, 16, 6, False), D.Dense(16, 4, D.SOFTMAX)],
    "block": [D.TransformerBlock(64, 2, 32, 128, False), D.Flatten(), D.Dense(2048, 4, D.SOFTMAX)],
    "embedding": [D.Embedding(30, 32, 8), D.TransformerBlock(32, 2, 8, 64, True), D.CLSPooling(8, 32), D.Dense(32, 4, D.LOGSOFTMAX)],
}


@pytest.mark.parametrize("kind", sorted(ANY_POINTER))
@pytest.mark.parametrize("batch", [5, 600])
def test_batches_at_any_float_address(device, kind, batch):
    """A batch in device memory may start at any float: the kernels that read it take their narrow loads there.  Against the same
    batch at the allocation's start, whose sums are the same."""
    from goneuron_b200.sequential import Adam, Sequential
    layers = ANY_POINTER[kind]
    rng = np.random.Generator(np.random.PCG64(4))
    params = configs.init_params(layers, rng)
    in_size = {"conv 5x5": 576, "conv 1x1": 256, "conv 3x3": 128, "pool": 192, "batch norm": 192, "dense": 64, "wide dense": 512, "lstm": 48, "gru": 48, "block": 2048, "embedding": 8}[kind]
    x = (rng.integers(0, 30, (batch, in_size)) if kind == "embedding" else rng.standard_normal((batch, in_size))).astype(np.float32)
    y = np.eye(4, dtype=np.float32)[rng.integers(0, 4, batch)]
    got = []
    for at in (0, 1):
        xd, yd = (device.alloc(np.concatenate([np.zeros(at, np.float32), a.ravel()])) for a in (x, y))
        model = Sequential(layers, device).Compile(Adam(1e-3), D.CROSS_ENTROPY)
        model.SetParams(params)
        loss = model.TrainBatchDevice(C.c_void_p(xd.value + 4 * at), C.c_void_p(yd.value + 4 * at), batch)
        got.append((loss, model.Gradients()))
        model.Close()
        device.free(xd); device.free(yd)
    assert abs(got[0][0] - got[1][0]) <= 1e-6 * max(1.0, abs(got[0][0]))
    assert norm_err(got[1][1], got[0][1]) <= 1e-6
