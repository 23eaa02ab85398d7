"""The work users have the framework do, as cases that can be timed: training steps and inference of `Sequential` models.

A case names a network builder of `goneuron_b200.configs` with its sizes and options, a batch, and how it is run:
"train" (`TrainBatch` on host arrays, as `Fit` calls it), "train_resident" (`TrainBatchDevice` on a batch that is already
in device memory) or "predict" (`PredictBatch`).  The sizes of the named configurations are the repository's benchmark
models; the others are generic, odd ones among them."""
import math

import numpy as np
import torch

from goneuron_b200 import configs
from goneuron_b200 import descriptors as D
from goneuron_b200.sequential import Adam, Device, Sequential

BUILDERS = {
    "mlp": configs.mlp,                  # Dense(ReLU) -> Dense(softmax)
    "mlp_act": configs.mlp_act,          # Dense(act) -> Dense(act) -> Dense(softmax)
    "cnn": configs.cnn,                  # (Conv2D -> MaxPool2D) x 2 -> Dense
    "cnn_bn": configs.cnn_bn,            # Conv2D -> BatchNorm2D -> MaxPool2D -> Dense
    "lstm": configs.recurrent,           # SequenceUnroller(LSTM) -> Dense
    "gru": configs.recurrent_gru,        # SequenceUnroller(GRU) -> Dense
    "transformer": configs.transformer,  # Embedding -> PositionalEncoding -> blocks -> CLSPooling -> Dense(log-softmax)
}
# make_inputs() goes by the layers; the learning rates are those of the benchmark configurations.  Transformers start
# with a warm-up, here the first of 4000 linear steps.
LEARNING_RATE = {"transformer": 3e-4 / 4000}


def listed():
    return [
        # one sample through the small classifier: a request of a service that answers them one by one; latency only
        dict(name="mlp_predict_1", net="mlp", mode="predict", batch=1, in_size=784, hidden=128, classes=10),
        # the MLP benchmark: a step of a few small layers, where launches and host work are what there is
        dict(name="mlp_train_64", net="mlp", mode="train", batch=64, in_size=784, hidden=128, classes=10),
        # tabular data: wide layers of odd sizes, a smooth activation, a batch that no tile divides
        dict(name="mlp_wide_train_1000", net="mlp_act", mode="train", batch=1000, in_size=333, hidden=1100, classes=37, act=D.GELU),
        # the CNN benchmark (32 x 32 colour images)
        dict(name="cnn_train_128", net="cnn", mode="train", batch=128, hw=32, c0=3, c1=16, c2=32, classes=10),
        # batch normalisation on grey 28 x 28 images, a ragged last batch of an epoch
        dict(name="cnn_bn_train_50", net="cnn_bn", mode="train", batch=50, hw=28, c0=1, c1=24, classes=10),
        # the recurrent benchmark: LSTM over 64 steps
        dict(name="lstm_train_256", net="lstm", mode="train", batch=256, in_size=16, hidden=128, seq_len=64),
        # a GRU on a batch that stays in device memory, odd sizes
        dict(name="gru_train_100", net="gru", mode="train_resident", batch=100, in_size=19, hidden=96, seq_len=50, return_seq=False),
        # the small language-model benchmark: causal, ReLU feed-forward, LayerNorm, head size 32
        dict(name="transformer_small_train_64", net="transformer", mode="train", batch=64, vocab=8192, dim=256, seq_len=128, heads=8,
             ff_dim=1024, n_blocks=4, ff_act=D.RELU, rms_norm=False, rope=False, causal=True),
        # an encoder that scores a few texts at once: bidirectional, forward only
        dict(name="encoder_predict_8", net="transformer", mode="predict", batch=8, vocab=8192, dim=512, seq_len=384, heads=8,
             ff_dim=2048, n_blocks=6, ff_act=D.RELU, rms_norm=False, rope=False, causal=False),
        # training an encoder classifier: bidirectional, GELU, a sequence length that no tile divides
        dict(name="encoder_train_24", net="transformer", mode="train", batch=24, vocab=5000, dim=384, seq_len=150, heads=12,
             ff_dim=1536, n_blocks=4, ff_act=D.GELU, rms_norm=False, rope=False, causal=False),
        # the block variants of newer models: SwiGLU, RMSNorm, rotary embeddings, head size 64
        dict(name="swiglu_train_16", net="transformer", mode="train", batch=16, vocab=8192, dim=512, seq_len=256, heads=8,
             ff_dim=1376, n_blocks=4, ff_act=D.SILU, rms_norm=True, rope=True, causal=False),
        # the large language-model benchmark, a quarter of its batch of 256 sequences
        dict(name="transformer_large_train_64", net="transformer", mode="train", batch=64, vocab=32000, dim=1024, seq_len=512, heads=16,
             ff_dim=4096, n_blocks=8, ff_act=D.RELU, rms_norm=False, rope=False, causal=True),
    ]


def _log(rng, lo, hi):
    """A whole number, spread evenly over the logarithm of lo .. hi."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _dense_tokens(c):
    return c["batch"] * c["seq_len"] * c["n_blocks"] * (4 * c["dim"] ** 2 + 3 * c["dim"] * c["ff_dim"] + c["seq_len"] * c["dim"])


def draw(rng):
    mode = rng.choice(["train", "train", "train_resident", "predict"])
    net = rng.choice(["mlp", "mlp_act", "cnn", "cnn_bn", "lstm", "gru", "transformer", "transformer", "transformer"])
    c = dict(net=net, mode=mode)
    if net in ("mlp", "mlp_act"):
        c.update(batch=_log(rng, 1, 2048), in_size=_log(rng, 16, 1024), hidden=_log(rng, 32, 2048), classes=_log(rng, 2, 200))
        if net == "mlp_act":
            c["act"] = rng.choice([D.GELU, D.SILU, D.TANH, D.SIGMOID])
    elif net in ("cnn", "cnn_bn"):
        c.update(batch=_log(rng, 4, 256), hw=4 * rng.randint(3, 10), c0=rng.choice([1, 3]), c1=rng.randint(6, 32), classes=_log(rng, 2, 100))
        if net == "cnn":
            c["c2"] = rng.randint(8, 64)
    elif net in ("lstm", "gru"):
        c.update(batch=_log(rng, 4, 256), in_size=_log(rng, 4, 64), hidden=rng.randint(16, 128), seq_len=_log(rng, 8, 64))
        if net == "gru":
            c["return_seq"] = rng.random() < 0.3
    else:
        limit = _dense_tokens(listed()[-1])
        while True:
            hd = rng.choice([32, 64, 64])
            c.update(batch=_log(rng, 1, 64), vocab=_log(rng, 500, 32000), seq_len=rng.choice([rng.randint(2, 32) * 16, _log(rng, 20, 512)]), heads=rng.randint(2, 16))
            c["dim"] = hd * c["heads"]
            c.update(ff_dim=c["dim"] * rng.choice([2, 3, 4]) + rng.choice([0, 0, 8, 36]), n_blocks=rng.randint(1, 8),
                     ff_act=rng.choice([D.RELU, D.GELU, D.SILU]), rms_norm=rng.random() < 0.3, rope=rng.random() < 0.3, causal=rng.random() < 0.5)
            if _dense_tokens(c) <= limit:
                break
    return c


_NOT_SIZES = ("name", "net", "mode", "batch")


def _layers(case):
    return BUILDERS[case["net"]](**{k: v for k, v in case.items() if k not in _NOT_SIZES})


class _Uniform:
    """Draws of the weight initialisers from a seeded generator on the GPU (quick for the large models)."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def uniform(self, lo, hi, size):
        return torch.empty(size, device="cuda").uniform_(lo, hi, generator=self.gen).cpu().numpy()


_device = None


class State:
    """A compiled model with its weights, and one batch."""

    def __init__(self, case, seed):
        global _device
        if _device is None:
            _device = Device(torch.cuda.current_device())
        layers, loss = _layers(case)
        self.mode, self.batch, self.resident = case["mode"], case["batch"], ()
        self.model = Sequential(layers, _device).Compile(Adam(LEARNING_RATE.get(case["net"], 1e-3)), loss)
        self.model.SetParams(configs.init_params(layers, _Uniform(seed)))
        self.x, self.y = configs.make_inputs(case["net"], layers, case["batch"], np.random.Generator(np.random.PCG64(seed)))
        if self.mode == "train_resident":
            self.resident = (_device.alloc(self.x), _device.alloc(self.y))

    def __del__(self):
        for p in self.resident:
            _device.free(p)
        if getattr(self, "model", None) is not None:
            self.model.Close()


class Trained(dict):
    """What a training step leaves behind.  Gradients, parameters and optimiser state stay in the model's device buffers,
    as in a training loop; an entry is read from there when it is looked up."""

    def __init__(self, state, loss):
        model, self.owner = state.model, state                  # the buffers live as long as their model
        super().__init__(loss=lambda: loss, gradients=model.Gradients, params=model.Params, adam=model.AdamState, layer_state=model.State)

    def __getitem__(self, key):
        return super().__getitem__(key)()


def prepare(case, seed):
    return State(case, seed)


def run(state):
    if state.mode == "predict":
        return state.model.PredictBatch(state.x)
    if state.mode == "train_resident":
        return Trained(state, state.model.TrainBatchDevice(*state.resident, state.batch))
    return Trained(state, state.model.TrainBatch(state.x, state.y))


def _block_work(l, B, last, train):
    """Parameters and operations of one TransformerBlock under a CLS pooling of token 0.  What reaches the pooled token, or
    a weight gradient, has to be computed and nothing else does: without a mask every token feeds the keys and values of
    the next block, but of the last block only token 0 is read, and in training the last token, whose activations are the
    input side of the inner layers' weight gradients.  With a causal mask token 0 sees itself alone, so inference needs
    only token 0, and so does the whole backward pass."""
    d, f, T = l.dim, l.ff_dim, l.seq_len
    n_ff = 3 if l.activation == D.SILU else 2
    P = 4 * (d * d + d) + (2 if l.kernel else 4) * d + n_ff * d * f + (0 if n_ff == 3 else f) + d
    nt = B * T
    if l.causal and not train:
        return P, 2.0 * B * (2 * d * d + n_ff * d * f)
    nq = B * (1 + (train and T > 1)) if last else nt
    pairs = B * (T + (1 if l.causal else T)) if last and train and T > 1 else B * T if last else B * (T * (T + 1) // 2 if l.causal else T * T)
    fl = 2.0 * (2 * nt * d * d + 2 * nq * d * d + n_ff * nq * d * f) + 4.0 * d * pairs
    if train:
        gq = B if last or l.causal else nt                      # tokens with a gradient behind the attention
        gk = B if l.causal else nt                              # ... and in front of it
        gp = B if l.causal else B * T if last else pairs
        fl += 2.0 * (n_ff * gq * d * f + 2 * gq * d * d + 2 * gk * d * d) + 8.0 * d * gp      # gradients of the activations
        fl += 2.0 * B * 4 * d * d + 2.0 * d * f * (B * n_ff if n_ff == 2 else B + 2 * gq)     # gradients of the weights
    return P, fl


def work(case):
    layers, _ = _layers(case)
    B, train = case["batch"], case["mode"] != "predict"
    P, fl, in_size = 0, 0.0, None
    for i, l in enumerate(layers):
        k, dx = l.kind, i > 0
        if k == D.DENSE:
            n, p = l.in_size * l.out_size, l.in_size * l.out_size + l.out_size
            fl += 2.0 * B * n * (1 + train * (1 + dx))
            size, out_size = l.in_size, l.out_size
        elif k == D.CONV2D:
            kk = l.kernel * l.kernel
            oh, ow = ((s + 2 * l.padding - l.kernel) // l.stride + 1 for s in (l.in_h, l.in_w))
            p = l.out_size * l.in_size * kk + l.out_size
            fl += 2.0 * B * oh * ow * l.out_size * l.in_size * kk * (1 + train * (1 + dx))
            size = l.in_size * l.in_h * l.in_w
        elif k == D.BATCHNORM2D:
            p = 2 * l.in_size
        elif k == D.LSTM_UNROLLED:
            H, n, bt = l.out_size, l.in_size, B * l.seq_len
            p = 4 * H * (n + H + 1)
            fl += 2.0 * bt * H * (n + H)                        # only the input gate's rows see the input and the state
            fl += train * 2.0 * bt * 4 * H * (H + n + H + 1)    # state gradient; rank-one updates of the clipped sum
            size = n * l.seq_len
        elif k == D.GRU_UNROLLED:
            H, n, bt = l.out_size, l.in_size, B * l.seq_len
            p = 3 * H * n + 2 * H * H + 3 * H
            fl += 2.0 * bt * (3 * H * n + 3 * H * H) + train * (2.0 * bt * 4 * H * H + 2.0 * B * 3 * H * n)
            size = n * l.seq_len
        elif k == D.EMBEDDING:
            p, size = l.in_size * l.out_size, l.seq_len
        elif k == D.POSENC:
            p = l.seq_len * l.dim
        elif k == D.TRANSFORMER_BLOCK:
            p, f = _block_work(l, B, layers[i + 1].kind == D.CLS_POOLING, train)
            fl += f
        else:
            p = 0
        P += p
        in_size = size if in_size is None else in_size
    if not train:
        read = P if layers[0].kind != D.EMBEDDING else P - layers[0].in_size * layers[0].out_size + B * layers[0].seq_len * layers[0].out_size
        return {"bytes": 4.0 * (B * (in_size + out_size) + read), "flops": fl}
    # batch in; parameters and both moments in and out, gradients out
    return {"bytes": 4.0 * (B * (in_size + out_size) + 7.0 * P), "flops": fl}


def tolerance(case):
    """Everything is 32-bit arithmetic.  Inference: rounding of sums of some thousand terms, through all layers.  Training:
    Adam divides by the root of the second moment, so that an element whose gradient is rounding noise moves by about the
    learning rate in a direction that nothing fixes (two steps of 1e-3 against weights of 0.02 to 0.1, in few elements), and
    a ReLU whose input is within rounding distance of zero opens or stays shut: one unit of one sample."""
    if case["mode"] == "predict":
        return {"rel": 1e-5, "max": 1e-3}
    if case["net"] == "transformer" and case["ff_act"] == D.RELU:
        return {"rel": 2e-3, "max": 0.5}
    return {"rel": 2e-4, "max": 0.2}
