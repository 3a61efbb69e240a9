"""General tables in class planes against the box-layout colour sweep: the same chains bit for bit
and the same energies, over linear and product colourings, boundaries, asymmetric tables (whose
energy needs every record) and the sizes where the classes are ragged."""
import numpy as np
import pytest

from nanomagmc_gb300 import _lib as L
from nanomagmc_gb300.sampler import Sampler, make_options, read_interactions

from general_tables import write_table

HALF_2D = [(2, -1), (2, 1), (2, -2), (1, 1), (1, 0), (1, -1), (1, -2), (0, 2)]          # 9 classes, product
HALF_3D = [(2, 2, 0), (2, 1, 0), (2, 0, 2), (2, -1, 0), (2, -1, -2), (2, -2, 0), (1, 2, 1), (1, 2, -1), (1, 0, 1),
           (1, -2, 2), (0, 2, 0), (0, 1, 1), (0, 1, 0), (0, 1, -2)]                      # 27 classes, product


def table(directory, name):
    """A named general table; "product2", "product3": +-offsets that need a product colouring;
    "one_way": records without their opposites."""
    if name in ("2d_j1j2", "2d_j1j3", "3d_j1j2"):
        return write_table(directory, name)
    half = {"product2": HALF_2D, "product3": HALF_3D, "one_way": [(1, 0), (0, 1), (1, 1), (2, -1)]}[name]
    path = "%s/%s.dat" % (directory, name)
    with open(path, "w") as f:
        for k, o in enumerate(half):
            for sign in ((1,) if name == "one_way" else (1, -1)):
                f.write(" ".join(str(sign * v) for v in o))
                f.write(" %.3f %.3f %.3f %.3f\n" % (0.2 + 0.05 * k, sign * 0.1, -sign * 0.02 * k, sign * 0.03))
    return path


def run(path, shape, edge, periodic, sign, half):
    dim = 3 if shape == "c" else 2
    opt = make_options(shape, edge=edge, periodic=periodic, J=1.0, D=0.5)
    s = Sampler(opt, read_interactions(path, dim, 1.0, 0.5), T=[0.5, 1.1, 2.0], H=[0.3, 0.0, -0.2], seed=4)
    s.option(L.OPT_HALF_KERNEL, half)
    s.option(L.OPT_DMI_SIGN, sign)
    colours = s.option(L.OPT_COLOURS)
    s.sweep(3)
    s.sweep(2, [2, 0])
    o1, q1 = s.sweep_measure(2)
    h, _ = s.sample(1, 2, with_q=True)
    o2, q2 = s.measure()
    spins = np.stack([s.get_spins(k) for k in range(3)])
    s.close()
    return spins, np.concatenate([o1[None], h, o2[None]]), np.stack([q1, q2]), colours


@pytest.mark.gpu
@pytest.mark.parametrize("sign", [0, 1])
@pytest.mark.parametrize("name,shape,edge,periodic", [
    ("2d_j1j2", "s", 12, True), ("2d_j1j2", "s", 10, False), ("2d_j1j3", "s", 30, True), ("2d_j1j3", "s", 14, False),
    ("3d_j1j2", "c", 8, True), ("3d_j1j2", "c", 10, False), ("3d_j1j2", "c", 16, True), ("product2", "s", 6, True),
    ("product2", "s", 12, True), ("product2", "s", 8, False), ("product3", "c", 6, True), ("product3", "c", 12, True),
    ("one_way", "s", 12, True), ("one_way", "s", 10, False)])
def test_class_planes_identical(tmp_path, name, shape, edge, periodic, sign):
    path = table(str(tmp_path), name)
    a, oa, qa, colours = run(path, shape, edge, periodic, sign, 0)
    b, ob, qb, _ = run(path, shape, edge, periodic, sign, 1)
    if name.startswith("product") and edge == 6:   # 12 has linear colourings of 12 classes
        assert colours in (9, 27)
    assert np.array_equal(a, b)
    N = edge ** (3 if shape == "c" else 2)
    # FP32 terms summed in another order: 2^-24 of at most 28 bonds of field 2 per site
    assert np.all(np.abs(oa - ob) <= 2.0 ** -24 * 64 * N)
    assert np.all(np.abs(qa - qb) <= 2.0 ** -20 * edge ** 2)
