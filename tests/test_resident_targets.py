"""On-chip runs of many sources with many targets each (blocks of a matrix of
Green's functions) against the step kernels: the same bits, and no slower."""
import numpy as np
import pytest

from test_resident import SCALE, _hermitian, _pair
from tbtk_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,K", [(1, 1), (2, 33), (5, 64), (16, 65), (33, 200), (64, 31), (128, 3)])
@pytest.mark.parametrize("N,complex_", [(31, True), (100, False), (513, True), (1800, False)])
def test_moments_bit_equal(gpu, N, complex_, B, K):
    """Targets in no order, some of them twice, rows with targets of many
    sources, blocks with up to and more than they stage."""
    r = np.random.default_rng(N + K)
    csr = _hermitian(N, 6, complex_, N)
    frm = r.integers(0, N, B)
    to, owner = r.integers(0, N, B * K), r.permutation(np.repeat(np.arange(B), K))
    to[: B * K // 3] = to[0]
    for precision in (gpu.FP64, gpu.MIXED):
        a, b = _pair(gpu, csr, B, precision, False)
        x, y = (m.moments_batched(frm, to, owner, 40, 1e-3, precision)[0] for m in (a, b))
        assert x.tobytes() == y.tobytes(), precision


@pytest.mark.parametrize("alpha", [0.0, 0.3])
@pytest.mark.parametrize("L,B,K", [(16, 64, 512), (30, 64, 512), (30, 16, 1800), (50, 64, 512)])
def test_no_slower_than_launched_steps(gpu, L, B, K, alpha):
    """Device time of the recursion by default and with launched steps (a
    handle with a wait bound of its own)."""
    csr = workloads.square_csr(L, L, J=0.5, W=2.0, alpha=alpha, seed=L)
    N = csr[0].size - 1
    frm = np.arange(B) * (N // B)
    to, owner = np.tile(np.arange(K) * (N // K), B), np.repeat(np.arange(B), K)
    ms = []
    for bound in (None, 1 << 22):
        m = gpu.Matrix.from_csr(*csr, SCALE)
        m.set_profiling(True)
        if bound:
            m.set_wait_limit(bound)
        best = np.inf
        for _ in range(3):
            m.moments_batched(frm, to, owner, 200, 1e-3, gpu.FP64)
            best = min(best, m.profile()[0])
        ms.append(best)
    assert ms[0] <= 1.2 * ms[1], ms
