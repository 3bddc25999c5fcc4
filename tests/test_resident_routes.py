"""Which calls run on chip and which as launched steps: an on-chip run adds a
handful of kernel launches, launched steps one and more each."""
import numpy as np
import pytest

from test_resident import SCALE, _hermitian
from tbtk_b200 import lattice as L

pytestmark = pytest.mark.gpu

M = 200  # 199 steps, or 100 with doubling


def _launches(gpu, call):
    n = gpu.kernel_launches()
    call()
    return gpu.kernel_launches() - n


def _ldos_launches(gpu, m, sites, precision):
    tab = gpu.Table.create(M, gpu.tbtk_range(-SCALE, SCALE, 20, False, False), SCALE)
    return _launches(gpu, lambda: m.ldos_sites(tab, sites, 1e-3, precision))


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("N,B", [(N, B) for N in (1, 31, 100, 513, 1800) for B in (1, 2, 12, 64, 128)
                                 if N < 1800 or B < 64])
def test_small_matrices_run_on_chip(gpu, N, B, complex_):
    """Sizes that test_resident compares with the step kernels (1800 randomly
    coupled rows of 64 and 128 FP64 sources are faster launched: 7.8 and 9.2 us a
    step against 12 and 24)."""
    m = gpu.Matrix.from_csr(*_hermitian(N, 6, complex_, N), SCALE)
    sites = (np.arange(B) * 5 % N).astype(np.uint32)
    for p in (gpu.FP64, gpu.MIXED, gpu.MIXED_DIRECT):
        assert _ldos_launches(gpu, m, sites, p) < 20, p
    n = _launches(gpu, lambda: m.moments_batched(sites, sites, np.arange(B), M, 1e-3, gpu.FP64))
    assert n < 20


@pytest.mark.parametrize("alpha", [0.0, 0.3])
def test_a_wait_bound_takes_launched_steps(gpu, alpha):
    """A handle with a wait bound runs the steps that have such waits, by
    default too; the bound of 0 gives up at once."""
    csr = L.square(24, 20, t=1.0, J=0.5, W=2.0, alpha=alpha, periodic=True, seed=5).csr()
    sites = np.arange(64, dtype=np.uint32)
    m = gpu.Matrix.from_csr(*csr, SCALE)
    m.set_fp64_head(0)
    assert _ldos_launches(gpu, m, sites, gpu.MIXED) < 20
    m.set_wait_limit(0)
    with pytest.raises(gpu.TBTKError) as e:
        _ldos_launches(gpu, m, sites, gpu.MIXED)
    assert e.value.status == gpu.ERR_TIMEOUT
    m.set_wait_limit(1 << 24)
    assert _ldos_launches(gpu, m, sites, gpu.MIXED) >= M // 2
    m.set_wait_limit()
    assert _ldos_launches(gpu, m, sites, gpu.MIXED) < 20


@pytest.mark.parametrize("side", [10, 30])
def test_tuning_sums_keeps_moments_on_chip(gpu, side):
    """Tuning the FP64 sums of a real matrix compares the vectors of doubles
    with the step kernels; its moment calls, on complex vectors, have a
    comparison of their own.  On chip wins both here (0.5 and 0.7 us a step
    against 3)."""
    csr = L.square(side, side, t=1.0, J=0.5, W=2.0, periodic=True, seed=side).csr()
    m = gpu.Matrix.from_csr(*csr, SCALE)
    m.autotune(4, gpu.FP64, ldos=True, probe_steps=64)
    sites = np.arange(4, dtype=np.uint32)
    assert _ldos_launches(gpu, m, sites, gpu.FP64) < 20
    assert _launches(gpu, lambda: m.moments_batched(sites, sites, sites, M, 1e-3, gpu.FP64)) < 20


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("alpha", [0.0, 0.3])
def test_saved_tuning_result_keeps_the_chip(gpu, alpha, precision):
    """What the autotuner returns for a small matrix, installed on a new
    handle, leaves its calls where tuning left them; another configuration
    makes them launched steps, until the default is installed again."""
    csr = L.square(30, 30, t=1.0, J=0.5, W=2.0, alpha=alpha, periodic=True, seed=3).csr()
    p, sites = getattr(gpu, precision), np.arange(4, dtype=np.uint32)
    m = gpu.Matrix.from_csr(*csr, SCALE)
    tuned = m.autotune(4, p, ldos=True, probe_steps=64)
    assert tuned[:3] in m.configs_for(4, p, True) and tuned[3] > 0
    assert _ldos_launches(gpu, m, sites, p) < 20
    fresh = gpu.Matrix.from_csr(*csr, SCALE)
    fresh.set_fp64_head(0)
    fresh.set_config(4, p, *tuned[:3], ldos=True)
    assert _ldos_launches(gpu, fresh, sites, p) < 20
    other = [c for c in fresh.configs_for(4, p, True) if 1 <= c[2] <= 4][0]
    fresh.set_config(4, p, *other, ldos=True)
    assert _ldos_launches(gpu, fresh, sites, p) >= M // 2
    fresh.set_config(4, p, 1, 4, 0, ldos=True)
    assert _ldos_launches(gpu, fresh, sites, p) < 20
    for bad in ((1, 8, 0), (2, 2, 0), (4, 1, 0)):
        with pytest.raises(gpu.TBTKError):
            fresh.set_config(4, p, *bad, ldos=True)
