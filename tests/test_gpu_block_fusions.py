"""Kernels and dispatch branches that take several passes of a TransformerBlock at once, at the sizes where they can go wrong:
norms with rows in registers, stacked projections and plane-writing epilogues on the tensor-core engine, contractions cut into
slices, outer products in 128-row tiles, and weight maxima left behind by the update."""
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


def _parity(device, oracle, layers, batch, kind="transformer", seed=7):
    from goneuron_b200.sequential import Adam, Sequential
    rng = np.random.Generator(np.random.PCG64(seed))
    params = configs.init_params(layers, rng)
    x, y = configs.make_inputs(kind, layers, batch, rng)
    ref = oracle.OracleState(layers, D.CROSS_ENTROPY, params, lr=1e-4)
    lit = oracle.OracleState(layers, D.CROSS_ENTROPY, params, lr=1e-4)
    loss_ref = ref.train_batch(x, y, W=2, threads=8, precision=64)
    lit.train_batch(x, y, W=2, threads=8, precision=32)
    model = Sequential(layers, device, virtual_workers=2).Compile(Adam(1e-4), D.CROSS_ENTROPY)
    model.SetParams(params)
    loss = model.TrainBatch(x, y)
    assert abs(loss - loss_ref) <= TOL * max(1.0, abs(loss_ref))
    assert_grads_close(layers, model.Gradients(), ref.grads, floor=lit.grads)
    model.Close()


@pytest.mark.parametrize("rows,n", [(1, 4), (9, 36), (300, 132), (17, 1000), (9, 1024), (2500, 96), (9, 1028), (9, 1026)])
def test_norm_rows_in_registers(device, rows, n):
    """Widths that fill part of a register row, the largest, and the first that do not fit; more rows than resident warps."""
    from goneuron_b200 import _lib
    rng = np.random.default_rng(rows + n)
    x = rng.standard_normal((rows, n)).astype(np.float32) * 2 + 0.3
    gamma, beta = rng.uniform(0.5, 1.5, n).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    dy = rng.standard_normal((rows, n)).astype(np.float32)
    y, dx, dg, db = np.empty_like(x), np.empty_like(x), np.empty(n, np.float32), np.empty(n, np.float32)
    _lib.check(_lib.load().gn_op_layernorm(device.handle, rows, n, _f(x), _f(gamma), _f(beta), _f(dy), _f(y), _f(dx), _f(dg), _f(db)))
    X, G, U = x.astype(np.float64), gamma.astype(np.float64), dy.astype(np.float64)
    xc = X - X.mean(1, keepdims=True); sd = np.sqrt((xc ** 2).mean(1, keepdims=True) + 1e-5); q = U * G
    assert norm_err(y, G * xc / sd + beta) <= TOL
    assert norm_err(dx, (q - q.sum(1, keepdims=True) / n) / sd - xc * (q * xc).sum(1, keepdims=True) / (n * sd ** 2)) <= TOL
    assert norm_err(dg, (U * xc / sd).sum(0)) <= TOL and norm_err(db, U.sum(0)) <= TOL


@pytest.mark.parametrize("kw", [dict(), dict(ff_act=D.GELU), dict(ff_act=D.SILU, rms_norm=True, rope=True), dict(ff_act=D.GELU, rms_norm=True)])
@pytest.mark.parametrize("T,dim,heads,ff", [(90, 192, 6, 416), (70, 224, 7, 388)])
def test_blocks_on_the_tensor_cores(device, oracle, T, dim, heads, ff, kw):
    """Rows and widths that are no multiples of a tile; the second width rules the plane-writing epilogues and the stacked gate
    and up matrices out (388 is no multiple of 32)."""
    layers = [D.Embedding(50, dim, T), D.PositionalEncoding(T, dim)] + [D.TransformerBlock(dim, heads, T, ff, c, **kw) for c in (False, True)]
    layers += [D.Flatten(), D.Dense(T * dim, 7, D.LOGSOFTMAX)]
    _parity(device, oracle, layers, 10)


@pytest.mark.parametrize("T,batch", [(5, 160), (31, 26), (32, 26), (33, 24)])
def test_plane_epilogue_gates_of_short_sequences(device, oracle, T, batch):
    """The plane-writing epilogue fetches the factors of two sequences per 32 rows ahead; sequences of fewer than 32 tokens have more, and a
    sequence's last row can lie anywhere in a warp's rows.  (GELU: its factors differ everywhere.)"""
    layers = [D.Embedding(50, 192, T), D.PositionalEncoding(T, 192)] + [D.TransformerBlock(192, 6, T, 416, False, D.GELU, False, False) for _ in range(2)]
    layers += [D.Flatten(), D.Dense(T * 192, 7, D.LOGSOFTMAX)]
    _parity(device, oracle, layers, batch)


@pytest.mark.parametrize("M,N,K", [(64, 352, 6000), (16, 100, 65600), (130, 65, 12000), (100, 1030, 1056)])
def test_contraction_in_slices(device, M, N, K):
    """Few output tiles and a long contraction: slices of 256 indices and up, a ragged last one, outputs with and without
    16-byte rows.  Bound: 2^-19 of sum |a b|: 2^-21 for the operands' 22 bits (three dropped terms of 2^-22 each), and as much again three times for the
    accumulator, which truncates once per 16 indices and term, and the partial sums in fp32."""
    from goneuron_b200 import _lib
    rng = np.random.default_rng(K)
    a, b, bias = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((N, K)).astype(np.float32), rng.standard_normal(N).astype(np.float32)
    c = np.empty((M, N), np.float32)
    _lib.check(_lib.load().gn_op_gemm_nt(device.handle, 1, M, N, K, _f(a), _f(b), _f(bias), _f(c)))
    ref = a.astype(np.float64) @ b.astype(np.float64).T + bias
    size = np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64).T
    assert np.max(np.abs(c - ref) / size) <= 2.0 ** -19


@pytest.mark.parametrize("batch,n_in,n_out", [(64, 1030, 2400), (3, 1030, 2400), (40, 130, 70)])
def test_outer_products(device, oracle, batch, n_in, n_out):
    """Weight and bias gradients of a Dense layer as a sum of a few outer products: 128- and 64-row tiles with ragged edges."""
    layers = [D.Dense(n_in, n_out, D.TANH), D.Dense(n_out, 5, D.LOGSOFTMAX)]
    _parity(device, oracle, layers, batch, kind="mlp")


def test_weight_maxima_from_the_update(device):
    """The planes of the weights are scaled by maxima that the previous step's update leaves behind; replacing the parameters by
    themselves makes the library find them anew.  Both must give the same bits."""
    from goneuron_b200.sequential import Adam, Sequential
    T, dim = 64, 96
    layers = [D.Embedding(41, dim, T), D.PositionalEncoding(T, dim)] + [D.TransformerBlock(dim, 3, T, 352, True, ff_act=a) for a in (D.RELU, D.SILU)]
    layers += [D.Flatten(), D.Dense(T * dim, 7, D.LOGSOFTMAX)]
    rng = np.random.Generator(np.random.PCG64(3))
    params = configs.init_params(layers, rng)
    x, y = configs.make_inputs("transformer", layers, 40, rng)
    got = []
    for again in (False, True):
        model = Sequential(layers, device).Compile(Adam(0.05), D.CROSS_ENTROPY)
        model.SetParams(params)
        losses = []
        for _ in range(5):
            losses.append(model.TrainBatch(x, y))
            if again:
                model.SetParams(model.Params())
        got.append((losses, model.Params().copy(), model.PredictBatch(x)))
        model.Close()
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1]) and np.array_equal(got[0][2], got[1][2])


@pytest.mark.parametrize("pool,masks", [(True, [True, True]), (True, [False, False]), (False, [True])])
def test_gradients_beside_the_main_stream(device, pool, masks):
    """Parameter gradients on the side stream (and in replayed graphs) against the same kernels one after the other, which is how a
    profiled model runs: same bits after several steps."""
    from goneuron_b200.sequential import Adam, Sequential
    T, dim, batch = 32, 256, 48
    layers = [D.Embedding(41, dim, T), D.PositionalEncoding(T, dim)] + [D.TransformerBlock(dim, 4, T, 512, c) for c in masks]
    layers += [D.CLSPooling(T, dim), D.Dense(dim, 600, D.LOGSOFTMAX)] if pool else [D.Flatten(), D.Dense(T * dim, 12, D.LOGSOFTMAX)]
    rng = np.random.Generator(np.random.PCG64(11))
    params = configs.init_params(layers, rng)
    x, y = configs.make_inputs("transformer", layers, batch, rng)
    got = []
    for profiled in (0, 1):
        model = Sequential(layers, device).Compile(Adam(1e-2), D.CROSS_ENTROPY)
        model.SetParams(params)
        model.set_profiling(profiled)
        got.append(([model.TrainBatch(x, y) for _ in range(6)], model.Params().copy()))
        model.Close()
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("R,N,K", [(40, 4200, 1040), (1000, 333, 1100), (4099, 256, 608), (12290, 96, 160)])
def test_weight_gradients_from_transposed_splits(device, oracle, R, N, K):
    """Dense weight gradients dZ^T X on the tensor cores: both operands are transposed on their way into planes.  One block per 32
    columns up to a full cluster, ragged rows and columns, rows without 16-byte alignment, and (the last) a contraction that does not
    fit the cluster's shared memory."""
    layers = [D.Dense(K, N, D.TANH), D.Dense(N, 3, D.LINEAR)]
    from goneuron_b200.sequential import Adam, Sequential
    rng = np.random.Generator(np.random.PCG64(R))
    params = configs.init_params(layers, rng)
    x, y = rng.standard_normal((R, K)).astype(np.float32), rng.standard_normal((R, 3)).astype(np.float32)
    model = Sequential(layers, device).Compile(Adam(1e-4), D.MSE)
    model.SetParams(params)
    model.TrainBatch(x, y)
    g = model.Gradients()
    model.Close()
    W1, b1 = params[:K * N].reshape(N, K).astype(np.float64), params[K * N:K * N + N].astype(np.float64)
    o = K * N + N
    W2, b2 = params[o:o + 3 * N].reshape(3, N).astype(np.float64), params[o + 3 * N:o + 3 * N + 3].astype(np.float64)
    X = x.astype(np.float64)
    a = np.tanh(X @ W1.T + b1)
    u = 2.0 * (a @ W2.T + b2 - y) / 3.0
    dz = (u @ W2) * (1.0 - a * a)
    for got, ref in ((g[:K * N].reshape(N, K), dz.T @ X), (g[K * N:o], dz.sum(0)), (g[o:o + 3 * N].reshape(3, N), u.T @ a)):
        assert norm_err(got, ref / R) <= TOL


@pytest.mark.parametrize("M,N", [(5, 130), (24, 5001), (32, 96), (70, 130)])
@pytest.mark.parametrize("K", [1, 31, 32, 33, 64, 65, 97, 500])
def test_cuda_core_contraction_steps(device, M, N, K):
    """One, two, three and more k-steps (two are in flight ahead of the one multiplied), ragged last ones, every tile shape.
    Bound: an fp32 sum of K products is within (K + 2) 2^-24 of sum |a b| + |bias|."""
    from goneuron_b200 import _lib
    rng = np.random.default_rng(M * 1000 + K)
    a, b, bias = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((N, K)).astype(np.float32), rng.standard_normal(N).astype(np.float32)
    c = np.empty((M, N), np.float32)
    _lib.check(_lib.load().gn_op_gemm_nt(device.handle, 0, M, N, K, _f(a), _f(b), _f(bias), _f(c)))
    ref = a.astype(np.float64) @ b.astype(np.float64).T + bias
    size = np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64).T + np.abs(bias)
    assert np.max(np.abs(c - ref) / size) <= (K + 2) * 2.0 ** -24


def test_cuda_core_contraction_of_millions_of_rows(device):
    """More tiles of 64 rows than a grid's second dimension has.  Bound as above."""
    from goneuron_b200 import _lib
    M, N, K = 65535 * 64 + 70, 8, 4
    rng = np.random.default_rng(1)
    a, b, bias = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((N, K)).astype(np.float32), rng.standard_normal(N).astype(np.float32)
    c = np.empty((M, N), np.float32)
    _lib.check(_lib.load().gn_op_gemm_nt(device.handle, 0, M, N, K, _f(a), _f(b), _f(bias), _f(c)))
    size = np.abs(a) @ np.abs(b).T + np.abs(bias)
    assert np.max(np.abs(c - (a.astype(np.float64) @ b.astype(np.float64).T + bias)) / size) <= (K + 2) * 2.0 ** -24
