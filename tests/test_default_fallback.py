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
