"""The generator's training arithmetic bit for bit: an Adam step divides a gradient by its own size and
rounds the weights to BF16, so that another rounding is a different training run a few steps on."""
import numpy as np
import pytest

from nanomagmc_gb300.warmstart import Generator, heisenberg_sampler

pytestmark = pytest.mark.gpu


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
