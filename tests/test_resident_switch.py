"""Batches around the sizes at which the recursion leaves the chip, several waves
of clusters among them: the bits of the launched steps (a handle with a wait
bound of its own runs those), and the default no slower than them."""
import numpy as np
import pytest

from conftest import rel_err
from test_fp64_head import cubic_csr
from test_resident import SCALE
from tbtk_b200 import lattice, workloads

pytestmark = pytest.mark.gpu


def _csr(name, L):
    if name == "honeycomb":
        return lattice.honeycomb(L, L, J=0.5, W=1.0, periodic=True, seed=4).csr()
    if name == "cubic":
        return cubic_csr(L, 1.0, 3)
    return workloads.square_csr(L, L, J=0.5, W=2.0, alpha=0.3 if name == "rashba" else 0.0, seed=L)


def _two(gpu, csr):
    a, b = (gpu.Matrix.from_csr(*csr, SCALE) for _ in range(2))
    b.set_wait_limit(1 << 22)
    return a, b


# 10k to 52k rows, odd sides among them
MODELS = [("square", 71), ("square", 103), ("square", 160), ("rashba", 77), ("rashba", 128),
          ("honeycomb", 50), ("honeycomb", 65), ("honeycomb", 90), ("cubic", 23), ("cubic", 30)]


@pytest.mark.parametrize("B", [1, 8, 17, 32, 64, 128])
@pytest.mark.parametrize("name,L", MODELS)
def test_equals_launched_steps(gpu, name, L, B):
    csr = _csr(name, L)
    sites = np.arange(B) * ((csr[0].size - 1) // B)
    a, b = _two(gpu, csr)
    for p in (gpu.FP64, gpu.MIXED):
        x, y = (m.moments_batched(sites, sites[::-1], np.arange(B), 40, 0.0, p)[0] for m in (a, b))
        assert np.array_equal(x, y), p
    tab = gpu.Table.create(90, gpu.tbtk_range(-SCALE, SCALE, 20, False, False), SCALE)
    x, y = (m.ldos_sites(tab, sites, 1e-3, gpu.FP64)[0] for m in (a, b))
    assert np.array_equal(x, y)
    x, y = (m.ldos_sites(tab, sites, 1e-3, gpu.MIXED)[0] for m in (a, b))
    assert rel_err(x, y) <= 1e-13  # regrouped FP64 sums


@pytest.mark.parametrize("name,L,B,precision", [
    ("honeycomb", 65, 48, "FP64"), ("honeycomb", 90, 128, "FP64"), ("square", 160, 8, "MIXED_DIRECT"),
    ("rashba", 90, 16, "MIXED"), ("rashba", 90, 32, "MIXED"), ("honeycomb", 90, 128, "MIXED_DIRECT"),
    ("square", 110, 128, "FP64"), ("cubic", 30, 48, "FP64"), ("rashba", 64, 8, "FP64"),
    ("square", 30, 1, "FP64"), ("square", 30, 64, "MIXED")])
def test_default_no_slower_than_launched_steps(gpu, name, L, B, precision):
    csr, p = _csr(name, L), getattr(gpu, precision)
    sites = np.arange(B) * ((csr[0].size - 1) // B)
    tab = gpu.Table.create(400, gpu.tbtk_range(-SCALE, SCALE, 8, False, False), SCALE)
    ms = []
    for m in _two(gpu, csr):
        m.set_fp64_head(0)
        m.set_profiling(True)
        best = np.inf
        for _ in range(5):
            m.ldos_sites(tab, sites, 1e-3, p)
            best = min(best, m.profile()[0])
        ms.append(best)
    assert ms[0] <= 1.2 * ms[1], ms
