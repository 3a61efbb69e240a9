"""nmmc_set_av_chains after a call that found no room for the sums: the same list again, once there is room."""
import numpy as np
import pytest

from nanomagmc_gb300 import _lib as L
from nanomagmc_gb300.sampler import Sampler, interactions_file, make_options, read_interactions

pytestmark = pytest.mark.gpu


def test_same_list_after_a_failed_allocation():
    """The sums of 2048 chains of 32^3 are 1.6 GB; all but 0.4 GB of the device is taken."""
    torch = pytest.importorskip("torch")
    n, edge = 2048, 32
    opt = make_options("c", edge=edge, periodic=True, J=1.0, D=0.3)
    s = Sampler(opt, read_interactions(interactions_file("3d_nn_bloch.dat"), 3, 1.0, 0.3), T=np.linspace(0.5, 2.0, n),
                H=0.1, seed=8)
    s.option(L.OPT_SWEEP_PATH, 1)
    s.sweep_measure(1)   # the path's scratch
    torch.cuda.init()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (400 << 20), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(L.NmmcError):
            s.set_av_chains(np.arange(n))
        with pytest.raises(L.NmmcError):   # nothing is summed
            s.get_av(0)
        s.sweep_measure(1, accumulate=True)
    finally:
        del filler
        torch.cuda.empty_cache()
    s.set_av_chains(np.arange(n))
    s.sweep_measure(1, accumulate=True)
    for k in (0, n - 1):
        assert np.array_equal(s.get_av(k), s.get_spins(k))
    s.close()
