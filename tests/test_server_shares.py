"""Tile-staged server steps over every share of tiles a block can get (none, a
part of a run, one run, several): results bit for bit those of the
register-staged steps, whose blocks take fixed runs and add per warp."""
import numpy as np
import pytest

from test_server import S, grid
from tbtk_b200 import workloads

pytestmark = pytest.mark.gpu


def _results(kpm, csrs, width, config, count=5):
    srv = kpm.Server(128, grid(), hbm_budget=8 << 30, tick_steps=32, tolerance=0)
    ids = [srv.add_model(*csr, S, width) for csr in csrs]
    srv.set_adaptive_width(False)
    if config:
        srv.set_config(width, *config)
    reqs = []
    for i, csr in zip(ids, csrs):
        N = csr[0].size - 1
        sites = np.unique(np.linspace(0, N - 1, min(width, count)).astype(np.uint32))
        reqs.append(srv.submit(i, sites, 100, 1e-3))
        if width > 8:
            reqs.append(srv.submit_greens(i, sites[:2], sites[:1].repeat(2), 60, 1e-3, "Retarded"))
    out = [srv.wait(r)[0] for r in reqs]
    srv.close()
    return out


@pytest.mark.parametrize("alpha", [0.0, 0.3])
@pytest.mark.parametrize("width", [4, 16, 64])
@pytest.mark.parametrize("sides", [[3], [97], [211], [430], [650], [3, 40, 97, 211, 64]])
def test_every_share_equals_register_staged(gpu, sides, width, alpha):
    csrs = [workloads.square_csr(L, L, t=1.0, J=0.5, W=2.0, alpha=alpha, seed=L) for L in sides]
    register = next(c for c in gpu.Server.step_configs(width, alpha == 0.0) if c[2] < 100000)
    for a, b in zip(_results(gpu, csrs, width, None),
                    _results(gpu, csrs, width, register)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("alpha", [0.0, 0.3])
@pytest.mark.parametrize("width", [1, 2])
@pytest.mark.parametrize("sides", [[3], [97], [430], [3, 40, 97, 211, 64]])
def test_narrow_lanes_equal_wider_ones(gpu, sides, width, alpha):
    """One and two lanes: register-staged, shorter runs on small models."""
    csrs = [workloads.square_csr(L, L, t=1.0, J=0.5, W=2.0, alpha=alpha, seed=L) for L in sides]
    register = next(c for c in gpu.Server.step_configs(4, alpha == 0.0) if c[2] < 100000)
    for a, b in zip(_results(gpu, csrs, width, None, width),
                    _results(gpu, csrs, 4, register, width)):
        assert np.array_equal(a, b)
