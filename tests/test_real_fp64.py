"""FP64 sums of a real matrix on vectors of doubles: the same values as the
complex128 recursion (set_real(False)), the reference's arithmetic."""
import numpy as np
import pytest

from tbtk_b200 import lattice as L

pytestmark = pytest.mark.gpu

SCALE, M, BROADENING = 12.0, 48, 1e-3


def _random_symmetric(N, per_row, seed):
    """A real symmetric CSR with ragged rows, some of them empty."""
    r = np.random.default_rng(seed)
    a = {}
    for _ in range(N * per_row // 2):
        i, j = (int(v) for v in r.integers(0, N, 2))
        if i % 7 == 3 or j % 7 == 3:
            continue
        a[i, j] = a[j, i] = float(r.uniform(-1, 1))
    rows = [[] for _ in range(N)]
    for (i, j), v in sorted(a.items()):
        rows[i].append((j, v))
    rowptr = np.cumsum([0] + [len(x) for x in rows]).astype(np.uint32)
    col = np.array([j for x in rows for j, _ in x], dtype=np.uint32)
    return rowptr, col, np.array([v for x in rows for _, v in x], dtype=np.complex128)


def _both(kpm, csr, B, scale=SCALE, configs=(None,)):
    """LDOS on complex vectors, and on real ones for each configuration."""
    N = csr[0].size - 1
    sites = (np.arange(B) * 37 % N).astype(np.uint32)
    tab = kpm.Table.create(M, kpm.tbtk_range(-scale, scale, 33, False, False), scale)
    m = kpm.Matrix.from_csr(*csr, scale)
    m.set_real(False)
    ref, _ = m.ldos_sites(tab, sites, BROADENING, kpm.FP64)
    out = []
    for c in configs:
        m = kpm.Matrix.from_csr(*csr, scale)
        if c is not None:
            m.set_config(B, kpm.FP64, *c)
        out.append(m.ldos_sites(tab, sites, BROADENING, kpm.FP64)[0])
    return ref, out


@pytest.mark.parametrize("B", [1, 2, 3, 4, 7, 16, 20, 64, 65, 128])
@pytest.mark.parametrize("N", [1, 63, 64, 257, 700])
def test_every_real_config_equals_complex(gpu, N, B):
    csr = _random_symmetric(N, 6, N)
    configs = [c for c in gpu.configs_for(B, gpu.FP64) if c[2] >= 200000000]
    assert configs
    ref, out = _both(gpu, csr, B, configs=[None] + configs)
    for o in out:
        assert np.array_equal(o, ref)


def test_large_single_source_equals_complex(gpu):
    """Above the size at which a single source takes real vectors by itself;
    an odd number of rows, whose last pair of staged rows is half empty."""
    csr = L.square(257, 261, t=1.0, J=0.0, W=2.0, seed=3).csr()
    N = 131073
    keep = int(csr[0][N])
    inside = csr[1][:keep] < N
    rowptr = np.concatenate([[0], np.cumsum(np.add.reduceat(inside, csr[0][:N].astype(np.int64)))])
    ref, out = _both(gpu, (rowptr.astype(np.uint32), csr[1][:keep][inside], csr[2][:keep][inside]), 1)
    assert np.array_equal(out[0], ref)


@pytest.mark.parametrize("B", [1, 2, 33])
def test_overflow_equals_complex(gpu, B):
    """A scale factor far below the spectrum: the recursion overflows, and the
    result is what the complex recursion gives."""
    csr = _random_symmetric(300, 6, 5)
    ref, out = _both(gpu, csr, B, scale=1e-8)
    assert not np.isfinite(ref).all()
    assert np.array_equal(out[0], ref, equal_nan=True)


def test_density_and_moments(gpu):
    """The density takes real vectors; moments keep the complex recursion and
    the signs of its zeros."""
    csr = _random_symmetric(400, 6, 9)
    e = gpu.tbtk_range(-SCALE, SCALE, 40, False, False)
    tab = gpu.Table.create(M, e, SCALE)
    sites = np.arange(5, 55, 5)
    res = []
    for real in (True, False):
        m = gpu.Matrix.from_csr(*csr, SCALE)
        m.set_real(real)
        mu, _ = m.moments_batched(sites, sites, np.arange(sites.size), M, 0.0, gpu.FP64)
        res.append((m.density(tab, sites, BROADENING, np.linspace(1, 0, 40), 0.6), mu))
    assert np.array_equal(res[0][0], res[1][0])
    assert res[0][1].tobytes() == res[1][1].tobytes()
