"""The on-chip recursion of small matrices against the step kernels: a batch
with a configuration of its own (set_config) runs those.  Stored vectors and
directly gathered moments agree bit for bit; the doubling sums are grouped
differently, so an LDOS from them agrees to the rounding of sums of N terms
below one (1e-13 of its maximum at N <= 6000)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

SCALE = 12.0


def _hermitian(N, per_row, complex_, seed, wide=0):
    """Hermitian CSR with ragged and empty rows; row 0 has `wide` entries."""
    r = np.random.default_rng(seed)
    a = {}
    pairs = [tuple(int(v) for v in r.integers(0, N, 2)) for _ in range(N * per_row // 2)]
    pairs += [(0, int(j)) for j in r.choice(N, size=wide, replace=False)]
    for i, j in pairs:
        if N > 8 and (i % 11 == 5 or j % 11 == 5):
            continue
        v = complex(r.uniform(-1, 1), r.uniform(-1, 1) if complex_ and i != j else 0.0)
        a[i, j], a[j, i] = v, v.conjugate()
    rows = [[] for _ in range(N)]
    for (i, j), v in sorted(a.items()):
        rows[i].append((j, v))
    rowptr = np.cumsum([0] + [len(x) for x in rows]).astype(np.uint32)
    col = np.array([j for x in rows for j, _ in x], dtype=np.uint32)
    return rowptr, col, np.array([v for x in rows for _, v in x], dtype=np.complex128)


def _pair(gpu, csr, B, precision, ldos):
    """The matrix by default, and with a step kernel for batches of B."""
    a, b = (gpu.Matrix.from_csr(*csr, SCALE) for _ in range(2))
    cfg = [c for c in b.configs_for(B, precision, ldos) if c[2] <= 4][0]
    b.set_config(B, precision, *cfg, ldos=ldos)
    return a, b


SIZES = [(1, 0), (31, 0), (33, 20), (100, 0), (513, 200), (1800, 0), (5000, 40)]


@pytest.mark.parametrize("B", [1, 2, 3, 12, 64, 128])
@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("N,wide", SIZES)
def test_moments_bit_equal(gpu, N, wide, complex_, B):
    csr = _hermitian(N, 6, complex_, N, min(wide, N))
    frm = (np.arange(B) * 7 % N).astype(np.uint32)
    for precision in (gpu.FP64, gpu.MIXED):
        for M in (1, 2, 3, 40):
            a, b = _pair(gpu, csr, B, precision, False)
            x, y = (m.moments_batched(frm, frm[::-1], np.arange(B), M, 0.0, precision)[0] for m in (a, b))
            assert x.tobytes() == y.tobytes(), (precision, M)


@pytest.mark.parametrize("B", [1, 2, 3, 12, 64, 128])
@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("N,wide", SIZES)
def test_ldos_equal(gpu, N, wide, complex_, B):
    csr = _hermitian(N, 6, complex_, N + 1, min(wide, N))
    sites = (np.arange(B) * 5 % N).astype(np.uint32)
    for head in (32, 0):
        for M in (1, 2, 7, 120):
            tab = gpu.Table.create(M, gpu.tbtk_range(-SCALE, SCALE, 50, False, False), SCALE)
            a, b = _pair(gpu, csr, B, gpu.MIXED, True)
            a.set_fp64_head(head)
            b.set_fp64_head(head)
            x, y = (m.ldos_sites(tab, sites, 1e-3, gpu.MIXED)[0] for m in (a, b))
            assert rel_err(x, y) <= 1e-13, (head, M)
            a, b = _pair(gpu, csr, B, gpu.FP64, True)
            x, y = (m.ldos_sites(tab, sites, 1e-3, gpu.FP64)[0] for m in (a, b))
            assert np.array_equal(x, y), M


@pytest.mark.parametrize("K", [64, 65, 500])
def test_many_targets_of_one_source(gpu, K):
    """More targets than a block stages, and a source of several columns."""
    csr = _hermitian(700, 6, True, 3)
    to = np.arange(K).astype(np.uint32)
    for owner, frm in ((np.zeros(K), [5]), (np.arange(K) % 3, [5, 9, 5])):
        a, b = _pair(gpu, csr, len(frm), gpu.FP64, False)
        x, y = (m.moments_batched(frm, to, owner, 60, 1e-3, gpu.FP64)[0] for m in (a, b))
        assert x.tobytes() == y.tobytes()


def test_several_launches(gpu):
    """More steps than one launch takes, with and without doubling sums."""
    csr = _hermitian(64, 4, False, 8)
    a, b = _pair(gpu, csr, 1, gpu.FP64, False)
    x, y = (m.moments(3, [3, 4], 9001, 0.0) for m in (a, b))
    assert x.tobytes() == y.tobytes()
    M = 35000
    tab = gpu.Table.create_clenshaw(M, gpu.tbtk_range(-SCALE, SCALE, 8, False, False), SCALE)
    sites = np.arange(128) % 64
    a, b = _pair(gpu, csr, 128, gpu.MIXED, True)
    x, y = (m.ldos_sites(tab, sites, 1e-4, gpu.MIXED)[0] for m in (a, b))
    assert rel_err(x, y) <= 1e-12


def test_autotune_keeps_the_faster(gpu):
    """After tuning a small matrix its calls are no slower than untuned."""
    csr = _hermitian(1800, 5, False, 4)
    m = gpu.Matrix.from_csr(*csr, SCALE)
    m.set_profiling(True)
    ms = []
    for tune in (False, True):
        if tune:
            t, v, mb, _ = m.autotune(4, gpu.MIXED, ldos=True, probe_steps=64)
            assert (t, v, mb) in m.configs_for(4, gpu.MIXED, True)
        tab = gpu.Table.create(512, gpu.tbtk_range(-SCALE, SCALE, 50, False, False), SCALE)
        times = []
        for _ in range(5):
            m.ldos_sites(tab, [1, 2, 3, 4], 1e-3, gpu.MIXED)
            times.append(m.profile()[0])
        ms.append(min(times[1:]))
    assert ms[1] <= 2 * ms[0]
