"""Tensor-core convolutions with the weights from their operand image against weights rearranged by the
threads: the same forward and data-gradient results bit for bit, at edges below and above a tile
row, with less than a tile per image and with many tiles per block."""
import numpy as np
import pytest

from nanomagmc_gb300.warmstart import Generator
from oracle import gen_oracle as G
from test_gpu_gen import small_dataset

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge,nimg", [(16, 1), (32, 17), (48, 5), (64, 1), (64, 40), (96, 3), (128, 2)])
@pytest.mark.parametrize("mode", [1, 3])
def test_weight_image_identical(edge, nimg, mode):
    gen = Generator(edge, 0, seed=4)
    gen.tensor_cores(mode)
    rng = np.random.default_rng(edge + nimg)
    x = G.bf16(np.maximum(rng.normal(size=(nimg, edge, edge, 48)), 0).astype(np.float32))
    for layer in (1, 6):
        gen.weight_image(True)
        a = gen.probe_conv(layer, x, True)
        gen.weight_image(False)
        assert np.array_equal(a, gen.probe_conv(layer, x, True))
    gen.close()


@pytest.mark.parametrize("edge", [32, 64])
def test_gradients_with_and_without_the_image(edge):
    out = []
    for on in (True, False):
        gen, _, _ = small_dataset(edge, 8)
        gen.weight_image(on)
        for step in range(2):   # the image follows the weights
            gen.train_step(np.arange(8), np.full(8, 0.3), 1e-3)
        out.append(np.asarray(gen.grads()).copy())
        gen.close()
    assert np.array_equal(out[0], out[1])
