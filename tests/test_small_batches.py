"""Every tile-staged form of small batches (rows of 4 to 32 bytes, staged four
columns at a time, and patterns of short runs) against the register-staged
steps: directly gathered moments bit for bit (zeros by value), doubling LDOS to
the rounding of its regrouped sums (1e-13 of its maximum)."""
import numpy as np
import pytest

from conftest import rel_err
from test_resident import SCALE, _hermitian
from tbtk_b200 import lattice as L

pytestmark = pytest.mark.gpu


def _models():
    yield "odd", _hermitian(523, 5, False, 1)
    yield "odd complex", _hermitian(521, 5, True, 2)
    yield "one tile", _hermitian(50, 4, False, 3)
    yield "honeycomb", L.honeycomb(9, 11, J=0.5, W=1.0, periodic=True, seed=4).csr()
    yield "wide rows", _hermitian(700, 40, False, 5)
    yield "wide complex rows", _hermitian(700, 30, True, 6)


MODELS = dict(_models())


@pytest.mark.parametrize("B", [1, 2, 3, 4, 8, 16, 33])
@pytest.mark.parametrize("name", list(MODELS))
def test_every_config_equals_register_staged(gpu, name, B):
    csr = MODELS[name]
    N, M = csr[0].size - 1, 24
    sites = (np.arange(B) * 13 % N).astype(np.uint32)
    tab = gpu.Table.create(M, gpu.tbtk_range(-SCALE, SCALE, 20, False, False), SCALE)
    for precision, ldos in ((gpu.FP64, False), (gpu.MIXED, False), (gpu.MIXED, True)):
        m = gpu.Matrix.from_csr(*csr, SCALE)
        configs = [c for c in m.configs_for(B, precision, ldos) if not 100 <= c[2] < 100000]
        register = [c for c in configs if c[2] <= 4][:1]
        ref = None
        for c in register + [c for c in configs if c[2] >= 100000]:
            m.set_config(B, precision, *c, ldos=ldos)
            if ldos:
                got = m.ldos_sites(tab, sites, 1e-3, precision)[0]
            else:
                got = m.moments_batched(sites, sites[::-1], np.arange(B), M, 0.0, precision)[0]
            if ref is None:
                ref = got
            elif ldos:
                assert rel_err(got, ref) <= 1e-13, c
            else:
                assert np.array_equal(got, ref), c


@pytest.mark.parametrize("M", [2, 3, 40, 300])
def test_grouped_reductions(gpu, M):
    """Doubling sums of many steps reduced by one launch, and of fewer."""
    csr = MODELS["odd"]
    tab = gpu.Table.create(M, gpu.tbtk_range(-SCALE, SCALE, 20, False, False), SCALE)
    for B in (1, 5, 128):
        sites = (np.arange(B) * 3 % 523).astype(np.uint32)
        m = gpu.Matrix.from_csr(*csr, SCALE)
        resident = m.ldos_sites(tab, sites, 1e-3, gpu.MIXED)[0]
        cfg = [c for c in m.configs_for(B, gpu.MIXED, True) if c[2] >= 100000][0]
        m.set_config(B, gpu.MIXED, *cfg)
        assert rel_err(m.ldos_sites(tab, sites, 1e-3, gpu.MIXED)[0], resident) <= 1e-13
