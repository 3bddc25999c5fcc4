"""The FP64 head on matrices whose rows do and do not fit its lists, at its
shortest lengths and with several launches of sources, against doubling runs
whose head is the whole recursion's FP64 moments."""
import numpy as np
import pytest

from conftest import rel_err
from test_resident import SCALE, _hermitian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [2, 3, 9, 32])
@pytest.mark.parametrize("N,per_row,complex_", [(60, 4, False), (400, 4, True), (700, 30, False), (700, 30, True),
                                                (5000, 5, False), (9000, 4, True)])
def test_head_moments_are_fp64(gpu, N, per_row, complex_, steps):
    """A run of M = 2 steps + 2 moments takes `steps` FP64 steps, so all but
    its last FP32 step is exact: its LDOS equals FP64's to a few float
    roundings of one step's sums (1e-7 of the maximum)."""
    csr = _hermitian(N, per_row, complex_, N + steps)
    M = 2 * steps + 2
    tab = gpu.Table.create(M, gpu.tbtk_range(-SCALE, SCALE, 30, False, False), SCALE)
    for B in (1, 5, 300):
        sites = (np.arange(B) * 7 % N).astype(np.uint32)
        m = gpu.Matrix.from_csr(*csr, SCALE)
        m.set_batch_width(gpu.MIXED, 256)
        m.set_fp64_head(steps)
        got = m.ldos_sites(tab, sites, 1e-3, gpu.MIXED)[0]
        assert rel_err(got, m.ldos_sites(tab, sites, 1e-3, gpu.FP64)[0]) <= 1e-7, B
