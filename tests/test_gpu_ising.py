"""Ising word kernels (four sites to a 32-bit word, tabulated acceptance limits) against the
one-site kernels: the same chains bit for bit and the same observables."""
import numpy as np
import pytest

from nanomagmc_gb300 import _lib as L
from nanomagmc_gb300.sampler import Sampler, interactions_file, make_options, read_interactions


def run(shape, edge, periodic, J, half, n=3):
    dim = 3 if shape == "c" else 2
    opt = make_options(shape, edge=edge, ising=True, periodic=periodic, J=1.0, D=0.0)
    inter = read_interactions(interactions_file("3d_nn_bloch.dat" if dim == 3 else "2d_nn.dat"), dim, 1.0, 0.0)
    for k in range(inter.n):
        inter.J[k] = J[k % len(J)]
    s = Sampler(opt, inter, T=np.linspace(0.3, 4.5, n), H=np.linspace(-0.4, 0.7, n), seed=9)
    s.option(L.OPT_SWEEP_PATH, 1)
    s.option(L.OPT_HALF_KERNEL, half)
    s.sweep(4)
    s.set_point(1, 2.2, 0.0)
    s.sweep(3, [n - 1, 1])
    obs = s.sweep_measure(2, with_q=False)
    out = np.stack([s.get_spins(k)[:, 0] for k in range(n)])
    s.close()
    return out, obs


@pytest.mark.gpu
@pytest.mark.parametrize("J", [[1.0], [-0.7, 0.3, 0.45], [0.0]], ids=["one", "mixed", "none"])
@pytest.mark.parametrize("shape,edge,periodic,n", [("s", 8, True, 3), ("s", 8, False, 3), ("s", 64, True, 300),
                                                   ("s", 96, False, 40), ("c", 8, True, 3), ("c", 16, False, 3),
                                                   ("c", 32, True, 12), ("c", 32, False, 150), ("c", 40, False, 4)])
def test_ising_words_identical(shape, edge, periodic, J, n):
    a, oa = run(shape, edge, periodic, J, 0, n)
    b, ob = run(shape, edge, periodic, J, 1, n)
    assert np.array_equal(a, b)
    # energies of up to 2*dim bonds per site, J in FP32 in the one-site kernel (2^-24 relative)
    assert np.all(np.abs(oa[:, 0] - ob[:, 0]) <= 2.0 ** -22 * 6 * edge ** (3 if shape == "c" else 2))
    assert np.array_equal(oa[:, 1:], ob[:, 1:])


@pytest.mark.gpu
def test_log_does_not_decrease_over_the_uniforms():
    """The tables' bisection needs log(u) monotone over the 2^23 uniforms: a chain of cold spins in
    a field has every limit K in range, so a sweep of one-site tests agrees at each k near K (the
    chains above); here the limits themselves are ordered in the temperature."""
    opt = make_options("s", edge=8, ising=True, periodic=True, J=1.0, D=0.0)
    inter = read_interactions(interactions_file("2d_nn.dat"), 2, 1.0, 0.0)
    acc = []
    for T in (0.5, 1.0, 2.0, 4.0):
        s = Sampler(opt, inter, T=[T] * 64, H=0.0, seed=3)
        s.option(L.OPT_SWEEP_PATH, 1)
        up = np.zeros((64, 3))
        up[:, 0] = 1.0
        for k in range(64):
            s.set_spins(k, up)
        s.sweep(1)
        acc.append(sum(int((s.get_spins(k)[:, 0] < 0).sum()) for k in range(64)))
        s.close()
    assert acc == sorted(acc)
