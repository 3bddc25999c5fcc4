"""The energy sums at the edges of their splits (vectors per thread, energies
per block, terms ahead, parts of a host call) against the oracle's sums over
the same table: bit for bit, the reference's order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,M,E", [(1, 1, 1), (1, 31, 33), (2, 32, 31), (3, 33, 64), (1, 127, 65), (5, 128, 100),
                                   (17, 129, 127), (64, 200, 500), (65, 161, 1000), (140, 96, 960),
                                   (33, 4099, 40)])
def test_sums_bit_equal(gpu, oracle, K, M, E):
    r = np.random.default_rng(K * M + E)
    energies = gpu.tbtk_range(-9.0, 9.0, max(E, 2))[:E]
    host = oracle.lookup_table(M, energies, 10.0)
    t = gpu.Table.upload(host)
    mu = r.standard_normal((K, M)) + 1j * r.standard_normal((K, M))
    ldos = t.ldos(mu)
    greens = [t.greens(mu, ty) for ty in range(4)]
    for k in sorted({0, K // 2, K - 1}):
        assert np.array_equal(ldos[k], oracle.ldos_table(host, mu[k]))
        for ty in range(4):
            assert np.array_equal(greens[ty][k], oracle.greens_table(host, ty, mu[k])), ty
