"""The FP64 head on matrices with one long row (a lead or an impurity coupled to
many sites): a row of the ball costs its own entries, not the longest row's,
and a long row inside the ball ends the head at the step before it."""
import time

import numpy as np
import pytest

from conftest import rel_err
from test_fp64_head import S, block_diag
from tbtk_b200 import workloads

pytestmark = pytest.mark.gpu

M, GRID = 66, 60  # 33 steps: 32 of the head and one more


def _star(spokes):
    """A hub coupled to `spokes` sites; the hub is the last row."""
    r = np.random.default_rng(spokes)
    t = r.uniform(-1, 1, spokes) / np.sqrt(spokes)
    rowptr = np.append(np.arange(spokes + 1), 2 * spokes).astype(np.uint32)
    col = np.append(np.full(spokes, spokes), np.arange(spokes)).astype(np.uint32)
    return rowptr, col, np.append(t, t).astype(complex)


def _hub_on(csr, site, spokes):
    """csr and a star whose hub is also coupled to `site`."""
    rowptr, col, val = block_diag(csr, _star(spokes))
    hub = rowptr.size - 2
    end = int(rowptr[site + 1])
    rowptr = rowptr.astype(np.int64)
    rowptr[site + 1:] += 1
    col = np.append(np.insert(col, end, hub), 0).astype(np.uint32)
    val = np.append(np.insert(val, end, 0.5), 0)
    # the hub's row takes `site` as its first column
    h = int(rowptr[hub])
    col[h + 1:], val[h + 1:] = col[h:-1].copy(), val[h:-1].copy()
    col[h], val[h] = site, 0.5
    rowptr[hub + 1:] += 1
    return rowptr.astype(np.uint32), col, val


def _ldos(gpu, csr, sites, precision=None, head=32):
    m = gpu.Matrix.from_csr(*csr, S)
    m.set_fp64_head(head)
    t = gpu.Table.create(M, workloads.open_grid(S, GRID), S)
    return m.ldos_sites(t, sites, 1e-3, gpu.MIXED if precision is None else precision)[0]


@pytest.mark.parametrize("alpha", [0.0, 0.3])
@pytest.mark.parametrize("spokes", [5, 9, 10, 11, 31, 32, 33, 3000])
def test_long_row_outside_the_ball(gpu, spokes, alpha):
    """The head of a source that never meets the long row is the one of its
    lattice alone, to the rounding of regrouped sums."""
    lat = workloads.square_csr(40, 36, J=0.5, W=2.0, alpha=alpha, seed=spokes)
    sites = np.array([0, 777, 1439], dtype=np.uint32)
    got = _ldos(gpu, block_diag(lat, _star(spokes)), sites)
    assert rel_err(got, _ldos(gpu, lat, sites)) <= 1e-13


@pytest.mark.parametrize("alpha", [0.0, 0.3])
@pytest.mark.parametrize("spokes", [5, 9, 10, 11, 40, 3000, 6143, 6144, 20000])
def test_long_row_inside_the_ball(gpu, spokes, alpha):
    """The hub two and more steps from the sources, its neighbours inside a
    head's rows, or far beyond them (rows above 6144 entries take no head):
    the result of the FP64 recursion."""
    csr = _hub_on(workloads.square_csr(40, 36, J=0.5, W=2.0, alpha=alpha, seed=3), 100, spokes)
    sites = np.array([100, 102, 300, csr[0].size - 2], dtype=np.uint32)
    ref = _ldos(gpu, csr, sites, gpu.FP64)
    got = _ldos(gpu, csr, sites)
    for k in range(sites.size):
        assert rel_err(got[k], ref[k]) <= 1e-6, k


def test_a_long_row_elsewhere_costs_nothing(gpu):
    """Wall time outside the recursion steps and the energy sums, most of it the
    head's: with 6000 entries walked for every row of the ball it is more than
    ten times that of the lattice alone, with a row's own entries 1.3 times."""
    lat = workloads.square_csr(80, 80, J=0.5, W=2.0, seed=1)
    took = []
    for csr in (lat, block_diag(lat, _star(6000))):
        m = gpu.Matrix.from_csr(*csr, S)
        t = gpu.Table.create(M, workloads.open_grid(S, GRID), S)
        m.set_profiling(True)
        best = np.inf
        for _ in range(6):
            t0 = time.perf_counter()
            m.ldos_sites(t, [3210], 1e-3, gpu.MIXED)
            wall = time.perf_counter() - t0
            rec, energy, _ = m.profile()
            best = min(best, 1e3 * wall - rec - energy)
        took.append(best)
    assert took[1] <= 4 * took[0], took
