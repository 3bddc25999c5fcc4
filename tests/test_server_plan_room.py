"""Server classes whose models stage their columns four at a time (runs of one or
two rows) and share a ring with models of wider rows: where such copies leave no
room for a ring, columns are staged one at a time and the class stays
tile-staged.  A wait bound of 0 tells the two apart: only tile-staged steps have
waits that it ends."""
import numpy as np
import pytest

from test_server import S, grid

pytestmark = pytest.mark.gpu


def _shifted(sites, shifts, seed, phase=0.0):
    """Four orbitals a site; the first and the third couple to those of the
    sites `shifts` away: runs of one column, in aligned groups of four."""
    r = np.random.default_rng(seed)
    rows = [{} for _ in range(4 * sites)]
    for i in range(4 * sites):
        rows[i][i] = complex(r.uniform(-1, 1))
    for i in range(sites):
        for d in shifts:
            for a in (0, 2):
                for b in (0, 2):
                    v = r.uniform(-1, 1) * np.exp(1j * phase)
                    p, q = 4 * i + a, 4 * ((i + d) % sites) + b
                    rows[p][q], rows[q][p] = v, v.conjugate()
    return _csr(rows)


def _band(N, reach, seed):
    """Rows of 2 reach + 1 entries next to each other."""
    r = np.random.default_rng(seed)
    rows = [{i: complex(r.uniform(-1, 1))} for i in range(N)]
    for i in range(N):
        for j in range(i + 1, min(i + reach + 1, N)):
            rows[i][j] = rows[j][i] = complex(r.uniform(-1, 1) / reach)
    return _csr(rows)


def _csr(rows):
    rowptr = np.cumsum([0] + [len(x) for x in rows]).astype(np.uint32)
    col = np.array([j for x in rows for j in sorted(x)], dtype=np.uint32)
    return rowptr, col, np.array([x[j] for x in rows for j in sorted(x)])


SHIFTS = [37, 111, 301]


@pytest.mark.parametrize("sites", [999, 1000])
def test_one_model_stays_tile_staged(gpu, sites):
    """64 real lanes: a stage of 64 rows takes 131 KB with groups of four of the
    six neighbours' columns, 90 KB with single ones, of the 116 KB that two
    stages leave each."""
    srv = gpu.Server(128, grid(), hbm_budget=1 << 30, tick_steps=8, tolerance=0)
    mid = srv.add_model(*_shifted(sites, SHIFTS, 1), S, 64)
    srv.set_adaptive_width(False)
    srv.set_fp64_head(0)
    srv.set_wait_limit(0)
    with pytest.raises(gpu.TBTKError) as e:
        srv.wait(srv.submit(mid, np.arange(0, 128, 2), 64, 1e-3))
    assert e.value.status == gpu.ERR_TIMEOUT
    srv.close()


@pytest.mark.parametrize("width", [4, 16, 64])
@pytest.mark.parametrize("models", ["one", "room", "mixed", "wide", "complex"])
def test_equals_register_staged(gpu, models, width):
    phase = 0.4 if models == "complex" else 0.0
    csrs = [_shifted(999, SHIFTS[: 2 if models == "mixed" else 3], 1, phase)]
    if models in ("mixed", "wide"):
        csrs.append(_band(1501, 17, 2))
    if models in ("room", "complex"):
        csrs.append(_shifted(501, SHIFTS[:1], 3, phase))
    out = []
    register = next(c for c in gpu.Server.step_configs(width, models != "complex") if c[2] < 100000)
    for config in (None, register):
        srv = gpu.Server(256, grid(), hbm_budget=1 << 30, tick_steps=16, tolerance=0)
        ids = [srv.add_model(*csr, S, width) for csr in csrs]
        srv.set_adaptive_width(False)
        if config:
            srv.set_config(width, *config)
        reqs = [srv.submit(i, np.linspace(0, csr[0].size - 2, width).astype(np.uint32), 200, 1e-3)
                for i, csr in zip(ids, csrs)]
        out.append([srv.wait(r)[0] for r in reqs])
        srv.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
