"""Recurrences at the edges of their layouts: units per thread group (32, 128, above), one or two samples per block, clipping groups of
128 updates with remainders, worker chunks that end inside a group; and the element-wise functions against float64."""
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


@pytest.mark.parametrize("net,I,H,T,batch,W,seq", [
    ("lstm", 3, 1, 5, 3, 1, False), ("lstm", 4, 31, 9, 5, 1, True), ("lstm", 5, 33, 4, 149, 1, False), ("lstm", 6, 127, 3, 300, 1, False),
    ("lstm", 6, 128, 2, 151, 3, False), ("lstm", 2, 129, 3, 4, 1, False), ("lstm", 2, 160, 2, 150, 1, False), ("lstm", 1, 224, 2, 3, 1, False),
    ("lstm", 300, 9, 3, 100, 1, False),                  # a gradient wider than one column tile of the clipping kernel
    ("lstm", 4096, 8, 8, 8, 1, False),                   # a single group whose Gram product over the inputs is cut into slices
    ("lstm", 7, 20, 64, 2, 1, False),                    # one whole group
    ("lstm", 7, 20, 43, 3, 1, False),                    # 129 updates: a group of one
    ("lstm", 7, 20, 40, 10, 1, False), ("lstm", 7, 20, 40, 10, 4, False), ("lstm", 7, 20, 13, 21, 10, False),      # several groups; short last chunks; more than eight chunks
    ("gru", 3, 1, 5, 3, 1, False), ("gru", 4, 33, 6, 149, 1, True), ("gru", 5, 97, 4, 7, 1, False), ("gru", 5, 128, 3, 150, 1, False), ("gru", 5, 129, 3, 6, 1, False),
    # blocks of 32 units, one or two samples a block, weights beyond the registers (97 units and more), widths that no 16-byte load divides, one step
    ("lstm", 3, 97, 1, 3, 1, False), ("lstm", 5, 96, 5, 150, 1, True), ("lstm", 5, 101, 4, 149, 1, True), ("lstm", 5, 64, 6, 149, 1, False), ("lstm", 5, 100, 2, 148, 1, False), ("lstm", 3, 2, 3, 150, 1, True),
    ("gru", 5, 64, 1, 2, 1, False), ("gru", 5, 96, 5, 150, 1, True), ("gru", 5, 63, 4, 149, 1, False), ("gru", 3, 2, 3, 150, 1, False),
])
def test_recurrent_parity(device, oracle, net, I, H, T, batch, W, seq):
    from goneuron_b200.sequential import Adam, Sequential
    cell = D.SequenceUnrollerLSTM if net == "lstm" else D.SequenceUnrollerGRU
    layers = [cell(I, H, T, seq), D.Dense(H * T if seq else H, 2, D.LINEAR)]
    rng = np.random.Generator(np.random.PCG64(H + T))
    params = configs.init_params(layers, rng)
    x, y = configs.make_inputs(net, layers, batch, rng)
    y *= 3                                               # gradients well above the clipping norm
    ref = oracle.OracleState(layers, D.MSE, params, lr=1e-3)
    lit = oracle.OracleState(layers, D.MSE, params, lr=1e-3)
    out = oracle.OracleState(layers, D.MSE, params).forward_batch(x, threads=4, precision=64)
    loss_ref = ref.train_batch(x, y, W=W, threads=4, precision=64)
    lit.train_batch(x, y, W=W, threads=1 if W == 1 else W, precision=32)
    model = Sequential(layers, device, virtual_workers=W).Compile(Adam(1e-3), D.MSE)
    model.SetParams(params)
    assert norm_err(model.PredictBatch(x), out) <= TOL
    loss = model.TrainBatch(x, y)
    assert abs(loss - loss_ref) <= TOL * max(1.0, abs(loss_ref))
    assert_grads_close(layers, model.Gradients(), ref.grads, floor=lit.grads)
    model.Close()


@pytest.mark.parametrize("scale,W,batch", [(1e-6, 1, 20), (1e-2, 1, 20), (1.0, 1, 20), (1e4, 1, 20), (1e4, 4, 20), ("early", 1, 20), ("early", 2, 20), ("late", 1, 20),
                                           (1e-6, 1, 160), (1e4, 1, 160), ("early", 1, 160), ("late", 1, 160), (1e-6, 40, 160), (1e4, 40, 160), ("early", 40, 160)])
def test_clipping_walk_starts_where_the_result_can_still_see(device, oracle, scale, W, batch):
    """800 updates in seven groups (four chunks of 200, two of 400), 6400 in fifty, forty chunks of 160: nothing is clipped, some of it is,
    the last dozens of updates decide the result, or one sample's do -- an early one, whose group has to be walked although later
    groups only add small updates, or one in the last group."""
    from goneuron_b200.sequential import Adam, Sequential
    layers = [D.SequenceUnrollerLSTM(7, 20, 40, False), D.Dense(20, 2, D.LINEAR)]
    rng = np.random.Generator(np.random.PCG64(5))
    params = configs.init_params(layers, rng)
    x, y = configs.make_inputs("lstm", layers, batch, rng)
    if isinstance(scale, str):
        y *= 1e-4
        y[2 if scale == "early" else batch - 1] *= 1e9
    else:
        y *= scale
    ref = oracle.OracleState(layers, D.MSE, params, lr=1e-3)
    lit = oracle.OracleState(layers, D.MSE, params, lr=1e-3)
    ref.train_batch(x, y, W=W, threads=4, precision=64)
    lit.train_batch(x, y, W=W, threads=min(W, 8), precision=32)
    model = Sequential(layers, device, virtual_workers=W).Compile(Adam(1e-3), D.MSE)
    model.SetParams(params)
    model.TrainBatch(x, y)
    assert_grads_close(layers, model.Gradients(), ref.grads, floor=lit.grads)
    model.Close()


def test_clipping_keeps_what_is_not_finite(device, oracle):
    """An infinite target in the first sample: its updates are lost in no way, however large the later ones are."""
    from goneuron_b200.sequential import Adam, Sequential
    layers = [D.SequenceUnrollerLSTM(7, 20, 40, False), D.Dense(20, 2, D.LINEAR)]
    rng = np.random.Generator(np.random.PCG64(6))
    params = configs.init_params(layers, rng)
    x, y = configs.make_inputs("lstm", layers, 20, rng)
    y *= 1e4
    y[0] = np.inf
    ref = oracle.OracleState(layers, D.MSE, params, lr=1e-3)
    ref.train_batch(x, y, threads=4, precision=64)
    model = Sequential(layers, device).Compile(Adam(1e-3), D.MSE)
    model.SetParams(params)
    model.TrainBatch(x, y)
    n = params.size - 42                                  # the LSTM's parameters
    assert np.isnan(ref.grads[:n]).all() and np.isnan(model.Gradients()[:n]).all()
    model.Close()


def test_elementwise_functions_are_rounded_once(device):
    """exp and tanh come out within 0.54 ulp of the float64 value (one rounding gives 0.5).  Sigmoid and SiLU add two and three float32
    operations; a relative error of 2^-24 each and 1.08 * 2^-24 from the exponential is at most 3.1 and 4.1 ulp of the result."""
    from goneuron_b200.sequential import Adam, Sequential
    rng = np.random.default_rng(3)
    x = np.concatenate([rng.uniform(-12, 12, 60000), rng.uniform(-1, 1, 20000), rng.uniform(-104, 104, 20000), 10.0 ** rng.uniform(-30, -1, 5000),
                        [0.0, -0.0, 0.17, 0.17000001, 9.0, 9.1, 10.0, 88.7, -87.4, -103.9]]).astype(np.float32).reshape(-1, 1)
    xd = x.astype(np.float64)
    sig = 1 / (1 + np.exp(-xd))
    ref = {D.TANH: (np.tanh(xd), 0.54), D.SIGMOID: (sig, 3.1), D.SILU: (xd * sig, 4.1), D.ELU: (np.where(xd > 0, xd, np.exp(np.minimum(xd, 0)) - 1), None)}
    for act, (want, ulps) in ref.items():
        model = Sequential([D.Dense(1, 1, act)], device).Compile(Adam(1e-3), D.MSE)
        model.SetParams(np.array([1.0, 0.0], np.float32))
        got = model.PredictBatch(x).astype(np.float64)
        model.Close()
        if ulps is None:                                 # exp(x) - 1 in float32: half an ulp of 1 for the exponential, and the subtraction's
            assert np.max(np.abs(got - want) / np.maximum(1.0, np.abs(want))) <= 1.3 * 2.0 ** -24
            continue
        ok = np.abs(want) > 1e-35                        # (below it the exponential inside is denormal)
        ulp = np.spacing(np.abs(want).astype(np.float32)).astype(np.float64)
        assert np.max(np.abs(got - want)[ok] / ulp[ok]) <= ulps, (act, np.max(np.abs(got - want)[ok] / ulp[ok]))
        assert np.max(np.abs(got - want)[~ok]) <= 1e-37
    # GELU (the function of the plane-writing epilogues too): 2^-23 |x|, what the reference's float32 order leaves, and below it on average
    gelu = lambda v: v / (1 + np.exp(-2 * np.sqrt(2 / np.pi) * (v + 0.044715 * v ** 3)))      # noqa: E731
    xg = np.concatenate([rng.uniform(-6, 6, 400000), rng.uniform(-1, 1, 200000), 10.0 ** rng.uniform(-30, -1, 5000), [9.0, -9.0, 12.0, -12.0, 40.0]]).astype(np.float32).reshape(-1, 1)
    model = Sequential([D.Dense(1, 1, D.GELU)], device).Compile(Adam(1e-3), D.MSE)
    model.SetParams(np.array([1.0, 0.0], np.float32))
    with np.errstate(over="ignore"):
        err = np.abs(model.PredictBatch(xg) - gelu(xg.astype(np.float64))) / np.abs(xg.astype(np.float64))
    assert np.max(err) <= 2.0 ** -23 and np.sqrt(np.mean(err[:400000] ** 2)) <= 2.0 ** -25, (np.max(err), np.sqrt(np.mean(err[:400000] ** 2)))
    ends = model.PredictBatch(np.array([[np.inf], [-np.inf], [np.nan], [50], [-50], [0.0], [-3e38]], np.float32)).ravel()
    assert ends[0] == np.inf and np.isnan(ends[1:3]).all() and np.array_equal(ends[3:], [50, 0, 0, 0])
    model.Close()
    model = Sequential([D.Dense(1, 1, D.TANH)], device).Compile(Adam(1e-3), D.MSE)
    model.SetParams(np.array([1.0, 0.0], np.float32))
    assert np.array_equal(model.PredictBatch(np.array([[np.inf], [-np.inf], [50], [-50]], np.float32)).ravel(), [1, -1, 1, -1])
    assert np.isnan(model.PredictBatch(np.array([[np.nan]], np.float32))).all()
    model.Close()


@pytest.mark.parametrize("W,batch", [(1, 224), (2, 448)])
def test_replayed_step_walks_what_its_updates_ask_for(device, W, batch):
    """Seventy groups per chunk.  One recorded step is replayed with targets after which everything is walked, the last groups are, and (two
    chunks) one chunk is walked as a whole; every gradient is that of a model whose first step, issued launch by launch, it is."""
    from goneuron_b200.sequential import Adam, Sequential
    layers = [D.SequenceUnrollerLSTM(7, 20, 40, False), D.Dense(20, 2, D.LINEAR)]
    rng = np.random.Generator(np.random.PCG64(6))
    params = configs.init_params(layers, rng)
    x, y = configs.make_inputs("lstm", layers, batch, rng)
    half = np.ones_like(y)
    half[: batch // 2] = 1e-6

    def make(p):
        m = Sequential(layers, device, virtual_workers=W).Compile(Adam(1e-3), D.MSE)
        m.SetParams(p)
        return m
    model = make(params)
    for scale in (1e4, 1e4, 1e-6, 1e4, 1e4 * half, 1e-6, 1e4):
        other = make(model.Params())
        t = (y * scale).astype(np.float32)
        assert model.TrainBatch(x, t) == other.TrainBatch(x, t)
        assert np.array_equal(model.Gradients(), other.Gradients())
        other.Close()
    model.Close()
