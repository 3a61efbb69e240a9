"""Calls that follow one another without a synchronisation against one long call: the same chain bit for bit
on every streaming path (the sweep counters that one call advances are read by the next one's
first launch), and observables of a sample step the same as those of separate calls."""
import numpy as np
import pytest

from nanomagmc_gb300 import _lib as L
from nanomagmc_gb300.sampler import Sampler, interactions_file, make_options, read_interactions

from general_tables import write_table

pytestmark = pytest.mark.gpu

CASES = {
    "four_site": dict(shape="c", edge=16, table="3d_nn_bloch.dat"),
    "one_site": dict(shape="c", edge=16, table="3d_nn_bloch.dat", half=1),
    "odd_rows": dict(shape="s", edge=10, table="2d_nn_interfacial.dat"),
    "compact": dict(shape="x", edge=30, size=10.0, periodic=False, table="3d_nn_bloch.dat"),
    "masked": dict(shape="w", edge=30, size=9.0, periodic=False, table="2d_nn_interfacial.dat", compact=1),
    "ising_words": dict(shape="c", edge=16, ising=True, table="3d_nn_bloch.dat"),
    "ising": dict(shape="s", edge=10, ising=True, table="2d_nn.dat"),
    "classes": dict(shape="c", edge=8, table="3d_j1j2"),
    "colours": dict(shape="c", edge=8, table="3d_j1j2", half=1),
}


def sampler(tmp_path, case, n):
    dim = 3 if case["shape"] in "cx" else 2
    ising = case.get("ising", False)
    table = case["table"]
    path = interactions_file(table) if table.endswith(".dat") else write_table(str(tmp_path), table)
    opt = make_options(case["shape"], edge=case["edge"], size=case.get("size"), ising=ising,
                       periodic=case.get("periodic", True), J=1.0, D=0.0 if ising else 0.4)
    s = Sampler(opt, read_interactions(path, dim, 1.0, 0.0 if ising else 0.4), T=np.linspace(0.5, 2.5, n),
                H=np.linspace(-0.2, 0.3, n), seed=21)
    s.option(L.OPT_SWEEP_PATH, 1)
    s.option(L.OPT_HALF_KERNEL, case.get("half", 0))
    if "compact" in case:
        s.option(L.OPT_MASKED_COMPACT, case["compact"])
    return s


@pytest.mark.parametrize("n", [1, 5])
@pytest.mark.parametrize("name", list(CASES))
def test_calls_in_a_row(tmp_path, name, n):
    a, b = sampler(tmp_path, CASES[name], n), sampler(tmp_path, CASES[name], n)
    a.sweep(1)
    b.sweep(1)
    a.sweep(40)
    for _ in range(40):
        b.sweep(1)
    for k in range(n):
        assert np.array_equal(a.get_spins(k), b.get_spins(k))
    h, q = a.sample(1, 12, with_q=True)
    rows = [b.sweep_measure(1, accumulate=True) for _ in range(12)]
    assert np.array_equal(h, np.stack([r[0] for r in rows]))
    assert np.array_equal(q, np.stack([r[1] for r in rows]))
    assert np.array_equal(a.accumulators(), b.accumulators())
    for k in range(n):
        assert np.array_equal(a.get_spins(k), b.get_spins(k))
    a.close()
    b.close()
