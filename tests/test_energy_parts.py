"""Energy sums of many vectors on the host: they go up in at most four parts,
each of which runs the whole chain of terms, and every vector's sums are those
it has alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,M,E", [(256, 4096, 8), (257, 1000, 33), (1024, 1000, 2), (65, 4096, 100), (5, 7, 3)])
def test_few_parts(gpu, K, M, E):
    tab = gpu.Table.create(M, gpu.tbtk_range(-2.0, 2.0, E, False, False), 2.0)
    rng = np.random.default_rng(K)
    mu = rng.normal(size=(K, M)) + 1j * rng.normal(size=(K, M))
    n = gpu.kernel_launches()
    out = tab.ldos(mu)
    assert gpu.kernel_launches() - n <= 4
    g = tab.greens(mu, 1)
    for k in {0, K // 4 - 1, K // 4, K // 2, K - 1}:
        assert np.array_equal(out[k], tab.ldos(mu[k:k + 1])[0])
        assert np.array_equal(g[k], tab.greens(mu[k:k + 1], 1)[0])
