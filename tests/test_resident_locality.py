"""On chip or launched steps for matrices whose neighbours are not near in row
order: loads from other blocks are scattered there and cost several times as
much."""
import numpy as np
import pytest

from test_resident import SCALE
from test_row_locality import KINDS, _call, _csr

pytestmark = pytest.mark.gpu


def _both(gpu, name, L, B):
    csr = _csr(name, L)
    a, b = (gpu.Matrix.from_csr(*csr, SCALE) for _ in range(2))
    for m in (a, b):
        m.set_fp64_head(0)
        m.set_profiling(True)
    b.set_wait_limit(1 << 22)  # launched steps
    return a, b, (np.arange(B) * ((csr[0].size - 1) // B)).astype(np.uint32)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("B", [1, 2, 8, 32, 128])
@pytest.mark.parametrize("name,L", [("random", 40), ("random", 75), ("random", 110), ("random", 150),
                                    ("random rashba", 40), ("random rashba", 75)])
def test_no_slower_than_launched_steps(gpu, name, L, B, kind):
    """Up to 3.3 times the launched steps without the locality in the estimate;
    with it at most 1.34 among 465 batches of such matrices."""
    a, b, sites = _both(gpu, name, L, B)
    ms = []
    for m in (a, b):
        best = np.inf
        for _ in range(4):
            _call(gpu, m, kind, sites)
            best = min(best, m.profile()[0])
        ms.append(best)
    assert ms[0] <= 1.45 * ms[1], ms


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("B", [1, 7, 33])
@pytest.mark.parametrize("name,L", [("random", 13), ("random", 40), ("random rashba", 31), ("random", 90)])
def test_equals_launched_steps(gpu, name, L, B, kind):
    a, b, sites = _both(gpu, name, L, B)
    x, y = (_call(gpu, m, kind, sites) for m in (a, b))
    if kind == "ldos_mixed":
        assert np.max(np.abs(x - y)) <= 1e-13 * np.max(np.abs(y))
    else:
        assert np.array_equal(x, y)
