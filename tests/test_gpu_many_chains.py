"""Observables of more chains than the side-by-side finish takes at once: each chain's are the same bits as in a
call on a few of them, for one and for many slices and blocks per slice."""
import numpy as np
import pytest

from nanomagmc_gb300 import _lib as L
from nanomagmc_gb300.sampler import Sampler, interactions_file, make_options, read_interactions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,edge,size,ising,n", [
    ("s", 4, None, False, 2000), ("s", 10, None, True, 1500), ("c", 6, None, False, 1200), ("c", 7, None, False, 900),
    ("x", 7, 2.2, False, 1300), ("c", 40, None, True, 700), ("s", 130, None, False, 650), ("c", 34, None, False, 620)])
def test_many_chains(shape, edge, size, ising, n):
    dim = 3 if shape in "cx" else 2
    D = 0.0 if ising else 0.4
    opt = make_options(shape, edge=edge, size=size, ising=ising, periodic=edge % 2 == 0 and shape != "x", J=1.0, D=D)
    table = ("3d_nn_bloch.dat" if dim == 3 else "2d_nn_interfacial.dat") if not ising else (
        "3d_nn_bloch.dat" if dim == 3 else "2d_nn.dat")
    s = Sampler(opt, read_interactions(interactions_file(table), dim, 1.0, D), T=np.linspace(0.5, 2.0, n), H=0.1, seed=3)
    s.option(L.OPT_SWEEP_PATH, 1)
    s.sweep(2)
    for fp64 in (0, 1):
        s.option(L.OPT_MEASURE_FP64, fp64)
        o, q = s.measure()
        pick = np.r_[0:5, n // 2:n // 2 + 300, n - 3:n]
        po, pq = s.measure(pick)
        assert np.array_equal(o[pick], po) and np.array_equal(q[pick], pq)
        assert np.allclose(q.sum(1), o[:, 13], rtol=1e-9, atol=1e-9)
    s.reset_accumulators()
    s.measure(accumulate=True)
    a = s.accumulators()
    s.reset_accumulators()
    s.measure(pick, accumulate=True)
    assert np.array_equal(a[pick], s.accumulators()[pick])
    s.close()
