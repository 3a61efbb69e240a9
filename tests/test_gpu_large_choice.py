"""The automatic path of lattices too large for the record kernel: how often it is timed, what its cache
entries are made of, and a device without room to put the chains aside."""
import numpy as np
import pytest

from nanomagmc_gb300 import _lib as L
from nanomagmc_gb300.sampler import Sampler, interactions_file, make_options, read_interactions

pytestmark = pytest.mark.gpu


def sampler(n, edge=28, path=0):
    opt = make_options("c", edge=edge, periodic=True, J=1.0, D=0.3)
    s = Sampler(opt, read_interactions(interactions_file("3d_nn_bloch.dat"), 3, 1.0, 0.3), T=np.linspace(0.5, 2.0, n),
                H=0.1, seed=8)
    s.option(L.OPT_SWEEP_PATH, path)
    return s


def entries(tmp_path):
    f = [p for p in tmp_path.rglob("*") if p.is_file()]
    return [line for p in f for line in p.read_text().splitlines() if "/" in line.split()[0]]


def test_shrinking_list_is_timed_a_few_times(tmp_path, monkeypatch):
    monkeypatch.setenv("NMMC_CACHE_DIR", str(tmp_path))
    a, b = sampler(40), sampler(40, path=1)
    for n in range(40, 0, -1):
        a.sweep(1, np.arange(n))
        b.sweep(1, np.arange(n))
    assert len(entries(tmp_path)) <= 8 + 4 * 3   # 1 .. 8 each, then four to a factor of two
    for k in (0, 17, 39):
        assert np.array_equal(a.get_spins(k), b.get_spins(k))
    a.close()
    b.close()


@pytest.mark.parametrize("key,value", [("OPT_HALF_KERNEL", 1), ("OPT_WAVE", 1), ("OPT_MEASURE_FP64", 1),
                                       ("OPT_CHARGE_PASS", 1), ("OPT_MEASURE_SITES", 4), ("OPT_L2_PREFETCH", 0)])
def test_other_settings_leave_no_cache_entry(tmp_path, monkeypatch, key, value):
    monkeypatch.setenv("NMMC_CACHE_DIR", str(tmp_path))
    s = sampler(4)
    s.option(getattr(L, key), value)
    s.sweep(1)
    assert entries(tmp_path) == []
    s.close()
    s = sampler(4)
    s.sweep(1)
    assert len(entries(tmp_path)) == 1
    s.close()


def test_first_sweep_without_room_for_a_copy(tmp_path, monkeypatch):
    """The chains are 0.8 GB; all but 0.4 GB of the device is taken before the first sweep."""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("NMMC_CACHE_DIR", str(tmp_path))
    n = 2048
    s, few = sampler(n, edge=32), sampler(3, edge=32, path=1)
    few.set_points([0, 1, 2], *zip(*[s.get_point(k) for k in (0, 1, 2)]))
    s.synchronize()
    torch.cuda.init()
    free = torch.cuda.mem_get_info()[0]
    filler = torch.empty(free - (400 << 20), dtype=torch.uint8, device="cuda")
    try:
        s.sweep(2)
    finally:
        del filler
        torch.cuda.empty_cache()
    few.sweep(2)
    for k in range(3):
        assert np.array_equal(s.get_spins(k), few.get_spins(k))
    s.close()
    few.close()
