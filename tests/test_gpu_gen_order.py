"""The generator's gradients bit for bit: an Adam step divides a gradient by its own size and rounds
the weights to BF16, so that another order of additions is a different training run a few steps
on. Digests of whole training steps, and the FMA weight gradient against its order in numpy."""
import json
import os
import sys

import numpy as np
import pytest

from nanomagmc_gb300 import _lib as L
from nanomagmc_gb300.warmstart import Generator, heisenberg_sampler

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))
from make_gen_grads import CASES, digests  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge,batch,mode", CASES)
def test_gradients_of_four_steps(edge, batch, mode):
    want = json.load(open(os.path.join(HERE, "golden", "gen_grads.json")))["%d_%d_%d" % (edge, batch, mode)]
    assert digests(edge, batch, mode) == want


@pytest.mark.parametrize("nimg", [1, 5])
def test_fma_weight_gradient_order(nimg):
    """A partial per 16 x 16 pixel tile and four images: multiply-adds over its images, rows and pixels; then
    the partials from the first to the last. A BF16 x FP32 product is exact in FP64, so rounding the FP64
    sum to FP32 is the fused operation (but for a double rounding in about one of 2^29)."""
    E, C = 32, 48
    rng = np.random.default_rng(nimg)
    x = np.maximum(rng.standard_normal((nimg, E, E, C)), 0).astype(np.float32)
    x = (x.view(np.uint32) & 0xFFFF0000).view(np.float32)
    d = rng.standard_normal((nimg, E, E, C)).astype(np.float32)
    gen = Generator(E, 0, seed=1)
    got = np.zeros((9, C, C), np.float32)
    L.check(L.load().nmmc_gen_probe_wgrad(gen.h, nimg, x.ctypes.data, d.ctypes.data, got.ctypes.data, 0))
    pad = np.pad(x, ((0, 0), (1, 1), (1, 1), (0, 0)), mode="wrap").astype(np.float64)
    tot = np.zeros((9, C, C), np.float32)
    for grp in range(0, nimg, 4):
        for ty in range(0, E, 16):
            for tx in range(0, E, 16):
                acc = np.zeros((9, C, C), np.float32)
                for im in range(grp, min(grp + 4, nimg)):
                    for y in range(ty, ty + 16):
                        for xx in range(tx, tx + 16):
                            win = pad[im, y:y + 3, xx:xx + 3].reshape(9, C, 1)
                            acc = (win * d[im, y, xx].astype(np.float64) + acc).astype(np.float32)
                tot = tot + acc
    assert np.array_equal(got, tot)


def test_adam_steps_bit_for_bit():
    """The update's operations in numpy: FP32 each, the two sums of moments fused (a product of two FP32 values
    is exact in FP64, and its FP64 sum rounded to FP32 is the fused operation but for a double
    rounding in about one of 2^29)."""
    f = np.float32

    def fma(a, b, c):
        return (np.float64(a) * np.float64(b) + np.float64(c)).astype(f)

    E, n = 32, 4
    rng = np.random.default_rng(3)
    T, B = rng.uniform(0.3, 1.5, n), rng.uniform(0.0, 1.0, n)
    s = heisenberg_sampler(E, 0.5, T, B, seed=2)
    s.sweep(5)
    gen = Generator(E, capacity=n, seed=9)
    gen.add_snapshots(s, np.arange(n), np.stack([T, B, np.full(n, 0.5)], 1))
    b1, b2, lr = f(0.9), f(0.999), f(1e-3)
    p = np.asarray(gen.params(), f)
    m, v = np.zeros_like(p), np.zeros_like(p)
    for step in range(1, 6):
        gen.train_step(np.arange(n), np.full(n, 0.1 * step), 1e-3)
        g = np.asarray(gen.grads(), f)
        m = fma(f(1) - b1, g, b1 * m)
        w = (f(1) - b2) * g
        v = fma(w, g, b2 * v)
        c1, c2 = f(1) - f(float(b1) ** step), f(1) - f(float(b2) ** step)
        p = p - lr * (m / c1) / (np.sqrt(v / c2) + f(1e-8))
        assert np.array_equal(np.asarray(gen.params(), f), p)
    s.close()
