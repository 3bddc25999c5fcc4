"""Server steps whose staged-row waits run out while copies are still in flight:
the requests fail with a timeout, nothing of the step is added anywhere, and the
device goes on to serve others."""
import numpy as np
import pytest

from test_server import S, grid
from tbtk_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha", [0.0, 0.3])
@pytest.mark.parametrize("width", [4, 16, 64])
@pytest.mark.parametrize("L", [20, 61, 150])
def test_timeouts_leave_the_device_usable(gpu, L, width, alpha):
    csr = workloads.square_csr(L, L, J=0.5, W=2.0, alpha=alpha, seed=L)
    sites = np.arange(0, 2 * width, 2)
    out = []
    for limit in (0, 0, 0, None):
        srv = gpu.Server(128, grid(), hbm_budget=1 << 30, tick_steps=8, tolerance=0)
        mid = srv.add_model(*csr, S, width)
        srv.set_adaptive_width(False)
        srv.set_fp64_head(0)
        if limit is None:
            out.append(srv.wait(srv.submit(mid, sites, 64, 1e-3))[0])
        else:
            srv.set_wait_limit(limit)
            with pytest.raises(gpu.TBTKError) as e:
                srv.wait(srv.submit(mid, sites, 64, 1e-3))
            assert e.value.status == gpu.ERR_TIMEOUT
        srv.close()
    tab = gpu.Table.create(64, grid(), S)
    m = gpu.Matrix.from_csr(*csr, S)
    m.set_fp64_head(0)
    ref = m.ldos_sites(tab, sites, 1e-3, gpu.FP64)[0]
    assert np.max(np.abs(out[0] - ref)) <= 1e-5 * np.max(np.abs(ref))
