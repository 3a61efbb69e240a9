"""nmmc_get_spins by way of the device and of the host: the spins that were set, and no large buffer that
stays behind."""
import numpy as np
import pytest

from nanomagmc_gb300.sampler import Sampler, interactions_file, make_options, read_interactions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge", [32, 150])   # FP64 boxes of 0.8 and 81 MB
@pytest.mark.parametrize("ising", [False, True])
def test_spins_come_back(edge, ising):
    torch = pytest.importorskip("torch")
    opt = make_options("c", edge=edge, ising=ising, periodic=True, J=1.0, D=0.0)
    s = Sampler(opt, read_interactions(interactions_file("3d_nn_bloch.dat"), 3, 1.0, 0.0), T=[1.0, 2.0], H=0.1, seed=8)
    rng = np.random.default_rng(edge)
    v = np.zeros((edge ** 3, 3))
    if ising:
        v[:, 0] = rng.choice([-1.0, 1.0], edge ** 3)
    else:
        v = rng.standard_normal((edge ** 3, 3)).astype(np.float32).astype(np.float64)
    s.set_spins(0, v)
    s.synchronize()
    torch.cuda.init()
    free = torch.cuda.mem_get_info()[0]
    base = s.get_spins(1)
    assert np.array_equal(s.get_spins(0), v)
    assert free - torch.cuda.mem_get_info()[0] <= 66 << 20   # in pages of 2 MB
    assert np.array_equal(s.get_spins(1), base)
    s.close()
