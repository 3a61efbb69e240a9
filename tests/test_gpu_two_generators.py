"""Generators of several edges in one process: each keeps working when another was used in between."""
import numpy as np
import pytest

from test_gpu_gen import small_dataset

pytestmark = pytest.mark.gpu


def test_generators_of_other_edges_in_between():
    def step(edge):
        gen, _, _ = small_dataset(edge, 4)
        gen.train_step(np.arange(4), np.full(4, 0.4), 1e-3)
        return gen, np.asarray(gen.grads()).copy()

    rng = np.random.default_rng(2)
    x = np.maximum(rng.standard_normal((2, 64, 64, 48)), 0).astype(np.float32)
    a, _ = step(64)
    want = a.probe_conv(3, x, True)
    others = [step(edge)[0] for edge in (32, 128, 16)]
    assert np.array_equal(a.probe_conv(3, x, True), want)
    a.train_step(np.arange(4), np.full(4, 0.3), 1e-3)
    for gen in others:
        gen.train_step(np.arange(4), np.full(4, 0.3), 1e-3)
        assert np.all(np.isfinite(gen.grads()))
    for gen in [a] + others:
        gen.close()
