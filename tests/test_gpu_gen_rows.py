"""The row-ring convolutions and weight gradients of the generator where runs of rows begin and
end: at image edges, with one row per block, in strips of a row, and where a run wraps around the
rings of row buffers and accumulators."""
import ctypes as C

import numpy as np
import pytest

from oracle import gen_oracle as G
from test_gpu_gen import small_dataset

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nimg", [3, 17])
@pytest.mark.parametrize("layer", [0, 3, 7])
def test_run_boundaries_do_not_show(layer, nimg):
    """An image's convolution does not depend on how the batch's rows are split into runs: images of
    a batch equal the same image alone (one row per block), bit for bit, as every output is the
    same MMAs in the same order."""
    from nanomagmc_gb300.warmstart import Generator
    gen = Generator(128, 0, seed=4)
    rng = np.random.default_rng(17 * layer + nimg)
    x = G.bf16(np.maximum(rng.normal(size=(nimg, 128, 128, 8 if layer == 0 else 48)), 0).astype(np.float32))
    got = gen.probe_conv(layer, x, True)
    for i in sorted({0, nimg // 2, nimg - 1}):
        assert np.array_equal(got[i:i + 1], gen.probe_conv(layer, x[i:i + 1], True))
    gen.close()


@pytest.mark.parametrize("L_edge,nimg", [(32, 11), (48, 3), (64, 5), (192, 1)])
def test_weight_gradient_blocks(L_edge, nimg):
    """Weight gradient against an FP64 sum, to 2e-5 of the terms' magnitudes (the BF16 hi + lo split's
    2^-18 plus FP32 accumulation): whole rows of 32 to 64 positions and strips of 64 (L = 192)."""
    from nanomagmc_gb300 import _lib as L
    from nanomagmc_gb300.warmstart import Generator
    gen = Generator(L_edge, 0, seed=4)
    rng = np.random.default_rng(L_edge)
    x = np.ascontiguousarray(G.bf16(np.maximum(rng.normal(size=(nimg, L_edge, L_edge, 48)), 0)), np.float32)
    d = np.ascontiguousarray(rng.normal(size=(nimg, L_edge, L_edge, 48)), np.float32)
    got = np.zeros((9, 48, 48), np.float32)
    L.check(L.load().nmmc_gen_probe_wgrad(gen.h, nimg, x.ctypes.data_as(C.c_void_p), d.ctypes.data_as(C.c_void_p),
                                          got.ctypes.data_as(C.c_void_p), 1))
    d64 = d.reshape(-1, 48).astype(np.float64)
    for tap in range(9):
        xs = np.roll(x, shift=(1 - tap // 3, 1 - tap % 3), axis=(1, 2)).reshape(-1, 48).astype(np.float64)
        ref, mag = xs.T @ d64, np.abs(xs).T @ np.abs(d64)
        assert np.all(np.abs(got[tap] - ref) <= 2e-5 * mag + 1e-30), (tap, np.max(np.abs(got[tap] - ref) / mag))
    gen.close()


@pytest.mark.parametrize("L_edge,n", [(16, 2), (32, 5), (128, 2)])
def test_gradients_against_the_fma_path(L_edge, n):
    """Weight and bias gradients of one step, per layer, against the FMA path on the same batch. The
    forward passes round a few activations to neighbouring BF16 values, so the bar is that of the
    tensor-core path against the oracle, 3e-2 (test_gradients_match_oracle)."""
    grads = []
    for tensor in (1, 0):
        gen, _, _ = small_dataset(L=L_edge, n=n)
        gen.tensor_cores(tensor)
        gen.train_step(np.arange(n, dtype=np.int32), np.linspace(0.2, 0.8, n).astype(np.float32), lr=0.0)
        grads.append(G.unpack(gen.grads().astype(np.float64)))
        gen.close()
    for (w1, b1), (w0, b0) in zip(*grads):
        assert np.linalg.norm(w1 - w0) <= 3e-2 * np.linalg.norm(w0)
        assert np.linalg.norm(b1 - b0) <= 3e-2 * np.linalg.norm(b0)
