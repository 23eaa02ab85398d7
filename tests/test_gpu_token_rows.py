"""Which tokens of a TransformerBlock are computed depends on the layers above it (CLSPooling reads token 0 only): parity with
the CPU checker where that rule changes the path -- one and two blocks, one token, causal and not, mixed, every feed-forward
variant, and models without CLSPooling, whose blocks run all tokens in both directions."""
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


def _model(T, dim, heads, ff, masks, pool, vocab=60, classes=11, **kw):
    layers = [D.Embedding(vocab, dim, T), D.PositionalEncoding(T, dim)]
    layers += [D.TransformerBlock(dim, heads, T, ff, c, **kw) for c in masks]
    layers += [D.CLSPooling(T, dim), D.Dense(dim, classes, D.LOGSOFTMAX)] if pool else [D.Flatten(), D.Dense(T * dim, classes, D.LOGSOFTMAX)]
    return layers


CASES = [
    (1, 32, 2, 48, [True, True], True, {}), (1, 32, 2, 48, [False], True, {}),                       # a single token
    (2, 32, 2, 48, [False, False], True, {}),                                                        # token 0 and the last one are all
    (37, 48, 3, 100, [True, True, True], True, {}), (37, 48, 3, 100, [False, False], True, {}),
    (37, 48, 3, 100, [True, False, True], True, {}), (37, 48, 3, 100, [False, True], True, {}),       # mixed masks
    (300, 40, 5, 64, [False, False], True, {}),                                                      # head size 8, more keys than threads
    (20, 600, 1, 64, [False], True, {}),                                                             # head size above the block width
    (21, 66, 6, 36, [False, False], True, {}),                                                       # head size 11: no 16-byte loads
    (24, 64, 2, 96, [True, True], True, dict(ff_act=D.SILU, rms_norm=True, rope=True)),
    (24, 64, 2, 96, [False, False], True, dict(ff_act=D.SILU, rms_norm=True, rope=True)),
    (24, 64, 2, 96, [True, True], True, dict(ff_act=D.GELU, rope=True)), (24, 64, 2, 96, [False], True, dict(ff_act=D.GELU)),
    (128, 128, 2, 256, [True, True], False, {}), (128, 128, 2, 256, [False], False, {}), (40, 64, 2, 96, [True, True], False, dict(rope=True)),
    (250, 250, 2, 502, [False], False, {}),                                                          # residuals and gates of rows that 16-byte accesses do not fit
    (24, 66, 2, 70, [True, True], True, {}), (24, 128, 2, 130, [True, True, True], True, {}),         # a block's weight gradients in one launch, odd tiles
]


@pytest.mark.parametrize("T,dim,heads,ff,masks,pool,kw", CASES)
def test_token_rows_parity(device, oracle, T, dim, heads, ff, masks, pool, kw):
    _parity(device, oracle, _model(T, dim, heads, ff, masks, pool, **kw))


@pytest.mark.parametrize("below", [[], [D.PositionalEncoding(6, 32)], [D.TransformerBlock(32, 2, 6, 48, True)], [D.TransformerBlock(32, 2, 6, 48, False)],
                                   [D.PositionalEncoding(6, 32), D.TransformerBlock(48, 3, 4, 40, True)]])
def test_sequences_of_another_shape_below(device, oracle, below):
    """The layers below a causal block under CLSPooling read the same 192 floats as tokens of another width: token 0 of the one is not
    token 0 of the other."""
    _parity(device, oracle, [D.Embedding(60, 32, 6)] + below + [D.TransformerBlock(24, 2, 8, 40, True), D.CLSPooling(8, 24), D.Dense(24, 11, D.LOGSOFTMAX)])


def test_more_sequences_than_a_grid_dimension_has_for_three_projections(device, oracle):
    """22 000 short sequences: the token sums of dQ, dK and dV are 66 000 rows of one launch's second dimension."""
    _parity(device, oracle, _model(2, 16, 1, 16, [False], False, classes=3), batch=22000)


def test_full_width_block_with_gradients_at_every_token(device, oracle):
    """The block of the large language model (width 1024, 16 heads of 64, 512 tokens, feed-forward 4096) under a head that reads all tokens:
    tcgen05 attention in both directions, plane-writing gradient epilogues, contractions over 4096.  (Seed: the first for which all ReLU
    decisions of the last tokens, which gate whole gradient rows, are more than 2.9e-4 standard deviations from zero.)"""
    layers = [D.Embedding(300, 1024, 512), D.PositionalEncoding(512, 1024), D.TransformerBlock(1024, 16, 512, 4096, False, D.RELU), D.Flatten(),
              D.Dense(512 * 1024, 3, D.LOGSOFTMAX)]
    _parity(device, oracle, layers, batch=2, seed=9102)


def _parity(device, oracle, layers, batch=3, seed=99):
    from goneuron_b200.sequential import Adam, Sequential
    rng = np.random.Generator(np.random.PCG64(seed))
    params = configs.init_params(layers, rng)
    x, y = configs.make_inputs("transformer", layers, batch, rng)
    ref = oracle.OracleState(layers, D.CROSS_ENTROPY, params, lr=1e-4)
    out = oracle.OracleState(layers, D.CROSS_ENTROPY, params).forward_batch(x, threads=3, precision=64)
    lit = oracle.OracleState(layers, D.CROSS_ENTROPY, params, lr=1e-4)
    loss_ref = ref.train_batch(x, y, W=2, threads=4, precision=64)
    lit.train_batch(x, y, W=2, threads=2, precision=32)
    model = Sequential(layers, device, virtual_workers=2).Compile(Adam(1e-4), D.CROSS_ENTROPY)
    model.SetParams(params)
    assert norm_err(model.PredictBatch(x), out) <= TOL
    loss = model.TrainBatch(x, y)
    assert abs(loss - loss_ref) <= TOL * max(1.0, abs(loss_ref))
    assert_grads_close(layers, model.Gradients(), ref.grads, floor=lit.grads)
    model.SetParams(params)
    assert norm_err(model.PredictBatch(x), out) <= TOL          # and inference after a training step
    model.Close()
