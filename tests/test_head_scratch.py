"""Device memory and results of the FP64 head of many sources."""
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, rel_err
from test_fp64_head import S
from tbtk_b200 import workloads

pytestmark = pytest.mark.gpu

ROWS = 6144  # of a source's ball

_CHILD = """
import sys
sys.path[:0] = [%r, %r]
import numpy as np, torch
from tbtk_b200 import kpm, workloads
B, alpha = int(sys.argv[1]), float(sys.argv[2])
csr = workloads.square_csr(200, 200, J=0.5, W=2.0, alpha=alpha, seed=1)
tab = kpm.Table.create(100, workloads.open_grid(12.0, 8), 12.0)
def used(head):
    m = kpm.Matrix.from_csr(*csr, 12.0)
    m.set_batch_width(kpm.MIXED, B)
    m.set_fp64_head(head)
    m.ldos_sites(tab, np.arange(B) * 300, 1e-3, kpm.MIXED)
    return m, torch.cuda.mem_get_info()[0]
used(0)[0].close()
a, before = used(0)
b, free0 = used(0)
c, free1 = used(32)
print((before - free0), (free0 - free1))
"""


@pytest.mark.parametrize("alpha,entry,vectors,width", [(0.0, 10, 0, 5), (0.3, 18, 48, 9)])
@pytest.mark.parametrize("B", [128, 256])
def test_scratch_of_a_call(gpu, B, alpha, entry, vectors, width):
    """A head's scratch holds the entries that the matrix's rows have (value and
    index), and the vectors of a complex matrix, for the sources that run at
    once, one on each of at most 148 SMs; 6 MB of jobs, results and
    granularity."""
    out = subprocess.run([sys.executable, "-c", _CHILD % (str(ROOT), str(ROOT / "tests")), str(B), str(alpha)],
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    handle, with_head = map(int, out.stdout.split()[-2:])
    assert with_head - handle <= min(B, 148) * ROWS * (entry * width + vectors) + 6e6


@pytest.mark.parametrize("width", [8, 9, 10, 11])
def test_rows_around_the_listed_width(gpu, width):
    """Matrices whose widest row is at, below and above what a head lists: more
    sources than one launch takes, real and complex, against FP64."""
    for alpha in (0.0, 0.3):
        rowptr, col, val = workloads.square_csr(24, 22, J=0.5, W=2.0, alpha=alpha, seed=width)
        N = rowptr.size - 1
        rows = [dict(zip(col[rowptr[i]:rowptr[i + 1]], val[rowptr[i]:rowptr[i + 1]])) for i in range(N)]
        have = max(map(len, rows))
        for k in range(max(width - have, 0)):
            rows[500][600 + 7 * k] = rows[600 + 7 * k][500] = 0.25
        rowptr = np.cumsum([0] + [len(r) for r in rows]).astype(np.uint32)
        csr = (rowptr, np.array([j for r in rows for j in sorted(r)], dtype=np.uint32),
               np.array([r[j] for r in rows for j in sorted(r)], dtype=complex))
        sites = np.arange(0, N, 6, dtype=np.uint32)
        m = gpu.Matrix.from_csr(*csr, S)
        m.set_batch_width(gpu.MIXED, 256)
        t = gpu.Table.create(100, workloads.open_grid(S, 40), S)
        ref, _ = m.ldos_sites(t, sites, 1e-3, gpu.FP64)
        got, _ = m.ldos_sites(t, sites, 1e-3, gpu.MIXED)
        assert max(rel_err(got[k], ref[k]) for k in range(sites.size)) <= 1e-6
