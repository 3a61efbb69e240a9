"""Observables read from page-locked memory and from the device: series longer than the room for their
samples, lists of chains, and calls that do not read them, against calls one by one."""
import numpy as np
import pytest

from nanomagmc_gb300 import _lib as L
from nanomagmc_gb300.sampler import Sampler, interactions_file, make_options, read_interactions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nsamples", [(1, 70), (7, 90), (546, 3), (547, 3), (600, 20), (5000, 9)])
@pytest.mark.parametrize("path", [0, 1])
def test_series_equal_single_calls(n, nsamples, path):
    def make():
        opt = make_options("s", edge=8, ising=True, periodic=True, J=1.0, D=0.0)
        s = Sampler(opt, read_interactions(interactions_file("2d_nn.dat"), 2, 1.0, 0.0), T=np.linspace(1.5, 3.0, n), H=0.1,
                    seed=4)
        s.option(L.OPT_SWEEP_PATH, path)
        return s

    a, b = make(), make()
    part = np.arange(n)[::2]
    for chains in (None, part):
        h, q = a.sample(2, nsamples, chains, with_q=True)
        for k in range(nsamples):
            o, p = b.sweep_measure(2, chains, accumulate=True)
            assert np.array_equal(h[k], o) and np.array_equal(q[k], p)
    L.check(b.lib.nmmc_measure(b.h, None, n, None, None, 1))   # left on the device
    a.measure(accumulate=True)
    assert np.array_equal(a.accumulators(), b.accumulators())
    assert np.array_equal(a.measure(part)[0], b.measure(part)[0])
    a.close()
    b.close()
