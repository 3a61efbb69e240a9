"""FP32 observables of Heisenberg boxes by place against the FP64 mode: boundaries, DMI structures, and
edges where a row is shorter than a warp, no multiple of four sites of a colour, odd (masked for
the sweeps), and more rows than one block takes."""
import numpy as np
import pytest

from nanomagmc_gb300 import _lib as L
from nanomagmc_gb300.sampler import Sampler, make_options, read_interactions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table,dim", [("2d_nn_interfacial.dat", 2), ("2d_nn_bloch.dat", 2), ("3d_nn_bloch.dat", 3)])
@pytest.mark.parametrize("edge,periodic", [(4, True), (5, False), (10, True), (10, False), (33, False), (66, True),
                                           (67, False), (131, False)])
def test_box_observables_match_fp64(table, dim, edge, periodic):
    """Each FP32 total is a sum of at most edge^dim terms, added 16 per thread and 32 per warp before FP64:
    within 32 x 2^-24 ~ 2e-6 of the sum of the terms' magnitudes (at most 8 per site for the
    energy, pi per triangle for the charge), here 1e-5 per site."""
    if dim == 3 and edge > 67:
        pytest.skip("2-D only")
    data = __file__.rsplit("/", 2)[0] + "/data/Js/" + table
    opt = make_options("c" if dim == 3 else "s", edge=edge, periodic=periodic, J=1.0, D=0.4)
    s = Sampler(opt, read_interactions(data, dim, 1.0, 0.4), T=[0.3, 1.5], H=[0.2, -0.1], seed=6)
    s.option(L.OPT_HALF_KERNEL, 1)
    s.sweep(3)
    o32, q32 = s.measure()
    s.option(L.OPT_MEASURE_FP64, 1)
    o64, q64 = s.measure()
    s.close()
    n = edge ** dim
    assert np.max(np.abs(np.asarray(o32, float) - o64)) <= 1e-5 * n
    assert np.max(np.abs(np.asarray(q32, float) - q64)) <= 1e-5 * edge ** 2
