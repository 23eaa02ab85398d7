"""The small-product kernel at the edges of its tiles (8, 16 and 32 rows by 32 columns), stages of 64 indices, chunks and clusters, with and
without 16-byte copies, against float64."""
import ctypes as C

import numpy as np
import pytest

from goneuron_b200 import _lib, configs, descriptors as D
from tests.parity import TOL, assert_grads_close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    from goneuron_b200.sequential import Device
    d = Device(0)
    yield d
    d.close()


def product(device, A, B, bias):
    f = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))
    out = np.empty((A.shape[0], B.shape[0]), np.float32)
    _lib.check(_lib.load().gn_op_gemm_nt(device.handle, 0, A.shape[0], B.shape[0], A.shape[1], f(A), f(B), f(bias), f(out)))
    return out


@pytest.mark.parametrize("N,K", [(17, 64), (32, 65), (33, 128), (100, 257), (256, 1024), (260, 191), (384, 1536), (1100, 333), (2047, 512), (37, 4099), (20, 8192)])
def test_rows_against_float64_and_the_same_in_every_batch(device, N, K):
    """A warp adds up K / 8 products at most, then come seven warps, at most three levels of chunks and the bias: every output is within
    (K / 8 + 16) 2^-24 of the sum of magnitudes.  Rows do not depend on how many there are, whatever tile and cluster that gives."""
    rng = np.random.Generator(np.random.PCG64(N + K))
    A = rng.standard_normal((140, K)).astype(np.float32)
    B = rng.standard_normal((N, K)).astype(np.float32)
    bias = rng.standard_normal(N).astype(np.float32)
    exact = A.astype(np.float64) @ B.astype(np.float64).T + bias
    bound = (np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64).T + np.abs(bias)) * (K / 8 + 16) * 2.0 ** -24
    whole = product(device, A, B, bias)
    assert np.all(np.abs(whole - exact) <= bound)
    for m in (1, 7, 8, 9, 16, 17, 32, 33, 65):
        assert np.array_equal(product(device, A[:m], B, bias), whole[:m]), m


@pytest.mark.parametrize("N", [1, 10, 16])
@pytest.mark.parametrize("K", [128, 513, 1100, 2048, 4704])
def test_few_columns_against_float64_and_the_same_in_every_batch(device, N, K):
    """Sixteen columns or fewer: one row per cluster of blocks, or four where there are many (from 593, 297, 149 and 75 rows on for clusters of one, two, four and eight), with one to three rows
    left over.  A thread adds up K / 256 products at most, then come five exchanges, eight warps, eight blocks and the bias."""
    rng = np.random.Generator(np.random.PCG64(N + K))
    A = rng.standard_normal((603, K)).astype(np.float32)
    B = rng.standard_normal((N, K)).astype(np.float32)
    bias = rng.standard_normal(N).astype(np.float32)
    exact = A.astype(np.float64) @ B.astype(np.float64).T + bias
    bound = (np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64).T + np.abs(bias)) * (K / 256 + 24) * 2.0 ** -24
    whole = product(device, A, B, bias)
    assert np.all(np.abs(whole - exact) <= bound)
    for m in (1, 2, 70, 74, 75, 148, 150, 296, 299, 592, 601, 602):
        assert np.array_equal(product(device, A[:m], B, bias), whole[:m]), m


@pytest.mark.parametrize("M,N,K", [(3001, 33, 72), (5000, 33, 65), (2050, 130, 65), (9001, 33, 130), (5000, 70, 130), (9001, 33, 260),      # one, two and four chunks per block
                                   (5000, 33, 128), (5000, 100, 191), (777, 70, 256), (300, 100, 512),                              # ... a chunk per block of two, four and eight
                                   (5000, 100, 256), (5000, 100, 512), (5000, 33, 512)])                                            # ... several per block of several
def test_many_rows_have_the_sums_of_few(device, N, K, M):
    """Many tiles go to a kernel of larger tiles, which adds up in the same order: the same bits, whatever clusters both take."""
    rng = np.random.Generator(np.random.PCG64(M + N + K))
    A = rng.standard_normal((M, K)).astype(np.float32)
    B = rng.standard_normal((N, K)).astype(np.float32)
    bias = rng.standard_normal(N).astype(np.float32)
    whole = product(device, A, B, bias)
    for rows in (slice(0, 70), slice(M // 2, M // 2 + 33), slice(M - 65, M)):
        assert np.array_equal(product(device, A[rows], B, bias), whole[rows])
    bound = (np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64).T + np.abs(bias)) * (K / 8 + 16) * 2.0 ** -24
    assert np.all(np.abs(whole - (A.astype(np.float64) @ B.astype(np.float64).T + bias)) <= bound)


@pytest.mark.parametrize("I,H,O,batch", [(64, 64, 64, 64), (65, 33, 17, 65), (100, 200, 40, 70), (31, 129, 18, 300), (784, 128, 20, 127), (36, 300, 24, 1000), (9, 70, 1, 256),
                                          (9, 200, 72, 2050), (9, 99, 256, 2050), (333, 1100, 20, 100)])      # many tiles
def test_dense_gradients(device, oracle, I, H, O, batch):
    """Input and weight gradients of Dense layers: the operands' other orders, and the bias gradients that come with them."""
    from goneuron_b200.sequential import Adam, Sequential
    layers = [D.Dense(I, H, D.TANH), D.Dense(H, O, D.LINEAR)]
    rng = np.random.Generator(np.random.PCG64(I + batch))
    params = configs.init_params(layers, rng)
    x = rng.standard_normal((batch, I)).astype(np.float32)
    y = rng.standard_normal((batch, O)).astype(np.float32)
    ref = oracle.OracleState(layers, D.MSE, params, lr=1e-3)
    loss_ref = ref.train_batch(x, y, threads=4, precision=64)
    model = Sequential(layers, device).Compile(Adam(1e-3), D.MSE)
    model.SetParams(params)
    loss = model.TrainBatch(x, y)
    assert abs(loss - loss_ref) <= TOL * max(1.0, abs(loss_ref))
    assert_grads_close(layers, model.Gradients(), ref.grads)
    model.Close()
