"""Packed (two sites per instruction) quad kernels against the one-site kernel: the same chain
bit for bit, over the DMI structures, boundary conditions and the smallest and odd row counts."""
import numpy as np
import pytest

from nanomagmc_gb300 import _lib as L
from nanomagmc_gb300.sampler import Sampler, interactions_file, make_options, read_interactions

KINDS = ["none", "general", "pairs", "axial"]


def table(dim, kind):
    """Axis table whose DMI vectors have the structure the kernels specialise on."""
    inter = read_interactions(interactions_file("3d_nn_bloch.dat" if dim == 3 else "2d_nn_bloch.dat"), dim, 1.0, 0.4)
    for k in range(inter.n):
        o = np.array(list(inter.offset[k])[:dim] + [0] * (3 - dim))
        a, step = int(np.argmax(np.abs(o))), int(o.sum())
        inter.J[k] = 1.0 + 0.25 * a
        for c in range(3):
            inter.D[k][c] = {"none": 0.0, "general": 0.1 * (k + 1) - 0.05 * c, "pairs": step * (0.3 - 0.1 * c + 0.05 * a),
                             "axial": step * 0.4 * (c == a)}[kind]
    return inter


def chains(shape, edge, periodic, kind, **options):
    dim = 3 if shape == "c" else 2
    opt = make_options(shape, edge=edge, periodic=periodic, J=1.0, D=0.0 if kind == "none" else 1.0)
    s = Sampler(opt, table(dim, kind), T=[0.4, 1.3], H=[0.3, -0.2], seed=5)
    for key, v in options.items():
        s.option(getattr(L, key), v)
    s.sweep(4)
    s.sweep(3, [1])
    out = np.stack([s.get_spins(k) for k in range(2)])
    s.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("sign", [0, 1])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("shape,edge,periodic", [("s", 8, True), ("s", 24, False), ("s", 40, True), ("c", 8, False),
                                                 ("c", 16, True), ("c", 24, True)])
def test_quad_half_sweep_identical(shape, edge, periodic, kind, sign):
    a = chains(shape, edge, periodic, kind, OPT_SWEEP_PATH=1, OPT_DMI_SIGN=sign, OPT_HALF_KERNEL=0)
    b = chains(shape, edge, periodic, kind, OPT_SWEEP_PATH=1, OPT_DMI_SIGN=sign, OPT_HALF_KERNEL=1)
    assert np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3, 40])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("shape,edge,periodic", [("s", 2, True), ("s", 6, False), ("s", 10, True), ("s", 64, True),
                                                 ("s", 130, True), ("c", 4, True), ("c", 6, False), ("c", 10, True),
                                                 ("c", 30, True), ("c", 32, False)])
def test_cluster_stencil_identical(shape, edge, periodic, kind, n):
    """One chain per cluster of 1 to 16 CTAs: chains and observables against the streaming path."""
    dim = 3 if shape == "c" else 2
    opt = make_options(shape, edge=edge, periodic=periodic, J=1.0, D=0.0 if kind == "none" else 1.0)
    res = []
    for path, stencil in ((0, 2), (1, 0)):
        s = Sampler(opt, table(dim, kind), T=np.linspace(0.4, 1.3, n), H=np.linspace(0.3, -0.2, n), seed=5)
        s.option(L.OPT_SWEEP_PATH, path)
        s.option(L.OPT_RESIDENT_STENCIL, stencil)
        s.sweep(3)
        s.sweep(2, [n - 1])
        o, q = s.sweep_measure(2, accumulate=True)
        h, hq = s.sample(1, 2, np.arange(n)[::-1], with_q=True)
        res.append((np.stack([s.get_spins(k) for k in range(n)]), np.concatenate([o[None], h]),
                    np.concatenate([q[None], hq]), s.accumulators()))
        s.close()
    (sa, oa, qa, aa), (sb, ob, qb, ab) = res
    assert np.array_equal(sa, sb)
    # FP32 terms in another order: 2^-24 per term of at most 4 (energy) or 1, pi per angle
    N = edge ** dim
    tol = np.full(14, 2.0 ** -20 * N)
    tol[13] = 2.0 ** -20 * N
    assert np.all(np.abs(oa - ob) <= tol)
    assert np.all(np.abs(qa - qb) <= 2.0 ** -20 * edge ** 2 + 1e-6)
    assert np.array_equal(aa[:, 0], ab[:, 0])
