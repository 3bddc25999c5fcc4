"""The step kernel of matrices whose neighbours are not near in row order: a tile
would need a copy for every entry, so the default there is the register-staged
step; lattices keep the tile-staged one."""
import numpy as np
import pytest

from test_resident import SCALE
from tbtk_b200 import lattice, workloads

pytestmark = pytest.mark.gpu

TILED = 100000  # variants from here on are tile-staged


def _csr(name, L):
    if name == "honeycomb":
        return lattice.honeycomb(L, L, J=0.5, W=1.0, periodic=True, seed=4).csr()
    rp, col, val = workloads.square_csr(L, L, J=0.5, W=2.0, alpha=0.3 if "rashba" in name else 0.0, seed=L)
    if "random" not in name:
        return rp, col, val
    n = rp.size - 1
    p = np.random.default_rng(L).permutation(n)
    rows, cols = p[np.repeat(np.arange(n), np.diff(rp.astype(np.int64)))], p[col]
    o = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return rp.astype(np.uint32), cols[o].astype(np.uint32), val[o]


def _call(gpu, m, kind, sites):
    n = np.arange(sites.size)
    if kind.startswith("moments"):
        return m.moments_batched(sites, sites, n, 97, 0.0, gpu.FP64 if kind == "moments_fp64" else gpu.MIXED)[0]
    tab = gpu.Table.create(194, gpu.tbtk_range(-SCALE, SCALE, 8, False, False), SCALE)
    return m.ldos_sites(tab, sites, 1e-3, gpu.FP64 if kind == "ldos_fp64" else gpu.MIXED)[0]


def _ms(gpu, m, kind, sites):
    m.set_fp64_head(0)
    m.set_wait_limit(1 << 22)  # launched steps, also of small matrices
    m.set_profiling(True)
    best = np.inf
    for _ in range(4):
        _call(gpu, m, kind, sites)
        best = min(best, m.profile()[0])
    return best


# the register-staged default (threads per row, values per thread) of a batch
REGISTERS = {
    "fp64": {1: (1, 1), 2: (2, 1), 4: (4, 1), 8: (8, 1), 64: (32, 2)},
    "real": {1: (1, 1), 2: (1, 2), 4: (1, 4), 8: (1, 8), 64: (8, 8)},
    "complex": {1: (1, 1), 2: (1, 2), 4: (1, 4), 8: (4, 2), 64: (8, 8)},
}


KINDS = ["ldos_fp64", "moments_fp64", "ldos_mixed", "moments_mixed"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("B", [1, 2, 4, 8, 64])
@pytest.mark.parametrize("name,L", [("random", 110), ("random", 250), ("random rashba", 110),
                                    ("random rashba", 220)])
def test_no_slower_than_register_staged(gpu, name, L, B, kind):
    """The bound is the most that the estimates were off in 2112 batches;
    without the rule these take up to 12 times as long."""
    csr = _csr(name, L)
    sites = (np.arange(B) * ((csr[0].size - 1) // B)).astype(np.uint32)
    a, b = (gpu.Matrix.from_csr(*csr, SCALE) for _ in range(2))
    p, ldos = gpu.FP64 if kind.endswith("fp64") else gpu.MIXED, kind.startswith("ldos")
    cls = "fp64" if p == gpu.FP64 else "complex" if "rashba" in name else "real"
    b.set_config(B, p, *REGISTERS[cls][B], 2, ldos=ldos)
    ms = [_ms(gpu, m, kind, sites) for m in (a, b)]
    assert ms[0] <= 1.5 * ms[1], ms


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("B", [1, 7, 32])
@pytest.mark.parametrize("name,L", [("random", 75), ("random rashba", 71), ("honeycomb", 90), ("square", 110)])
def test_default_equals_tile_staged(gpu, name, L, B, kind):
    """The bits of a tile-staged step (1e-13 for sums that it groups)."""
    csr = _csr(name, L)
    sites = (np.arange(B) * ((csr[0].size - 1) // B)).astype(np.uint32)
    a, b = (gpu.Matrix.from_csr(*csr, SCALE) for _ in range(2))
    for m in (a, b):
        m.set_fp64_head(0)
        m.set_wait_limit(1 << 22)
    p, ldos = gpu.FP64 if kind.endswith("fp64") else gpu.MIXED, kind.startswith("ldos")
    cfg = [c for c in b.configs_for(B, p, ldos) if c[2] >= TILED][0]
    b.set_config(B, p, *cfg, ldos=ldos)
    x, y = (_call(gpu, m, kind, sites) for m in (a, b))
    if kind == "ldos_mixed":
        assert np.max(np.abs(x - y)) <= 1e-13 * np.max(np.abs(y))
    else:
        assert np.array_equal(x, y)
