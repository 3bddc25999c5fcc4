"""Where the tiles of a default do not fit the shared memory, the default takes
smaller tiles of the same threads and values per row."""
import numpy as np
import pytest

from test_resident import SCALE
from test_row_locality import _call, _csr, _ms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["ldos_fp64", "moments_fp64"])
@pytest.mark.parametrize("name,L,B", [("rashba", 130, 32), ("rashba", 250, 20), ("rashba", 250, 32)])
def test_same_shape_in_smaller_tiles(gpu, name, L, B, kind):
    """32 FP64 sources in 32-row tiles of 16 threads and 2 values do not fit
    two ring stages on a Rashba lattice, 16-row ones do; the tiles of 32
    threads took 1.2 to 1.4 times as long.  Timing noise is below 5%."""
    csr = _csr(name, L)
    sites = (np.arange(B) * ((csr[0].size - 1) // B)).astype(np.uint32)
    a, b = (gpu.Matrix.from_csr(*csr, SCALE) for _ in range(2))
    b.set_config(B, gpu.FP64, 16, 2, 116082, ldos=kind.startswith("ldos"))
    ms = [_ms(gpu, m, kind, sites) for m in (a, b)]
    assert ms[0] <= 1.1 * ms[1], ms
    assert np.array_equal(_call(gpu, a, kind, sites), _call(gpu, b, kind, sites))



@pytest.mark.parametrize("kind", ["moments_fp64"])
@pytest.mark.parametrize("L", [160, 254])
def test_better_tiles_without_locality(gpu, L, kind):
    """64 complex FP64 sources on randomly numbered square sites: smaller tiles
    of another shape halve the copies in a block's way.  Estimates are within
    a quarter in nine of ten batches."""
    csr = _csr("random", L)
    sites = (np.arange(64) * ((csr[0].size - 1) // 64)).astype(np.uint32)
    a, b = (gpu.Matrix.from_csr(*csr, SCALE) for _ in range(2))
    b.set_config(64, gpu.FP64, 16, 4, 108082, ldos=False)
    ms = [_ms(gpu, m, kind, sites) for m in (a, b)]
    assert ms[0] <= 1.3 * ms[1], ms


def _band(N, reach):
    i = np.repeat(np.arange(N), 2 * reach + 1)
    j = i + np.tile(np.arange(-reach, reach + 1), N)
    i, j = i[(j >= 0) & (j < N)], j[(j >= 0) & (j < N)]
    rp = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=N))])
    return rp.astype(np.uint32), j.astype(np.uint32), 0.2 * np.cos(i + j) + 0j


@pytest.mark.parametrize("kind", ["ldos_fp64", "moments_fp64"])
@pytest.mark.parametrize("N,B,config", [(20000, 1, (1, 1)), (20000, 2, (2, 1)), (60001, 1, (1, 1))])
def test_wide_rows_build_no_plans(gpu, N, B, config, kind):
    """Rows of 31 entries leave one or two FP64 sources no ring: the first call
    by default launches what it does with the register-staged step set."""
    csr = _band(N, 15)
    sites = (np.arange(B) * (N // B)).astype(np.uint32)
    n = []
    for c in (None, config):
        m = gpu.Matrix.from_csr(*csr, SCALE)
        m.set_wait_limit(1 << 22)  # launched steps
        if c:
            m.set_config(B, gpu.FP64, *c, 2, ldos=kind.startswith("ldos"))
        n.append(-gpu.kernel_launches())
        _call(gpu, m, kind, sites)
        n[-1] += gpu.kernel_launches()
    assert n[0] == n[1]
