"""Ising lattices that were given empty sites (spin 0) through nmmc_set_spins: observables and chains of the
word kernels against the one-site kernels and numpy."""
import numpy as np
import pytest

from nanomagmc_gb300 import _lib as L
from nanomagmc_gb300.sampler import Sampler, interactions_file, make_options, read_interactions

pytestmark = pytest.mark.gpu


def sampler(dim, edge, periodic, half):
    opt = make_options("c" if dim == 3 else "s", edge=edge, ising=True, periodic=periodic, J=1.0, D=0.0)
    s = Sampler(opt, read_interactions(interactions_file("3d_nn_bloch.dat" if dim == 3 else "2d_nn.dat"), dim, 1.0, 0.0),
                T=[1.5, 2.5, 4.0], H=[0.0, 0.2, -0.1], seed=12)
    s.option(L.OPT_SWEEP_PATH, 1)
    s.option(L.OPT_HALF_KERNEL, half)
    return s


@pytest.mark.parametrize("dim,edge,periodic", [(2, 16, True), (2, 40, False), (3, 8, True), (3, 32, True), (3, 16, False)])
def test_empty_sites(dim, edge, periodic):
    a, b = sampler(dim, edge, periodic, 0), sampler(dim, edge, periodic, 1)
    rng = np.random.default_rng(edge)
    v = np.zeros((edge ** dim, 3))
    v[:, 0] = rng.choice([-1.0, 0.0, 1.0], edge ** dim)
    for s in (a, b):
        s.sweep(2)
        s.set_spins(1, v)
    assert np.array_equal(a.get_spins(1), v)
    lat = v[:, 0].reshape((edge,) * dim)
    e = 0.0
    for axis in range(dim):
        nb = np.roll(lat, -1, axis)
        if not periodic:
            nb[tuple(slice(None) if k != axis else -1 for k in range(dim))] = 0.0
        e -= (lat * nb).sum()
    H = a.get_point(1)[1]
    for s in (a, b):
        o, _ = s.measure()
        assert o[1, L.OBS_E] == pytest.approx(e - H * lat.sum(), abs=1e-9 * lat.size)
        assert o[1, 1] == lat.sum()
    for k in range(4):   # sites fill as proposals are accepted
        oa, ob = a.sweep_measure(1), b.sweep_measure(1)
        assert np.array_equal(oa[0], ob[0])
        for c in range(3):
            assert np.array_equal(a.get_spins(c), b.get_spins(c))
    a.fork(1, 2)
    b.fork(1, 2)
    a.sweep(3, [2])
    b.sweep(3, [2])
    assert np.array_equal(a.get_spins(2), b.get_spins(2))
    v[:, 0] = rng.choice([-1.0, 1.0], edge ** dim)   # and none empty again
    for s in (a, b):
        for c in range(3):
            s.set_spins(c, v)
        s.sweep(3)
    for c in range(3):
        assert np.array_equal(a.get_spins(c), b.get_spins(c))
    a.close()
    b.close()
