"""CSR x SparseSign at the row count from which a lane takes a row alone (one call of
exactly that many rows, one more, and a tile and a row more), and with every
SKEMA_SSIGN_BATCH on both sides, against the FP64 oracle. Bar: 1e-6, a row's few
dozen terms."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import rel_fro

pytestmark = pytest.mark.gpu


def _check(oracle, m, n, rank, nu, calls):
    import torch

    import skema_b200 as sk

    rng = np.random.default_rng(m)
    cnt = rng.integers(0, 12, size=m)
    cnt[m // 2] = n // 2
    row = np.repeat(np.arange(m), cnt)
    A = sp.csr_matrix((rng.normal(size=row.size), (row, rng.integers(0, n, row.size))), shape=(m, n))
    A.sum_duplicates()
    A.data = A.data.astype(np.float32).astype(np.float64)
    a = sk.AlgParams(matrix_m=m, matrix_n=n, rank=rank, window=m, sketch_nu=nu, issparse=True, dim_redux=1)
    o = oracle.OracleSketch(m, n, rank, m, kind=1, issparse=True, nu=nu)
    o.reset()
    t = (torch.from_numpy(A.indptr.astype(np.int64)).cuda(), torch.from_numpy(A.indices).cuda(),
         torch.from_numpy(A.data.astype(np.float32)).cuda())
    with sk.SketchySVD(a) as s:
        s.reset()
        for _ in range(calls):
            s.update_rows(t, 0)
            o.update_rows(A, 0, m)
        for name, g, want in zip("XYZ", s.get_sketches(), (o.X, o.Y, o.Z)):
            assert rel_fro(g, want) < 1e-6, name


@pytest.mark.parametrize("rank", [20, 50])
@pytest.mark.parametrize("past", [0, 1, 9])
@pytest.mark.parametrize("calls", [1, 2])
def test_at_the_line(lib_built, oracle, rank, past, calls):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _check(oracle, 8 * sms * (1024 // (4 * rank + 1)) + past, 300, rank, 0.9, calls)


@pytest.mark.parametrize("batch", [2, 4, 6, 8])
@pytest.mark.parametrize("m", [700, 6100])
def test_batches(lib_built, oracle, monkeypatch, batch, m):
    monkeypatch.setenv("SKEMA_SSIGN_BATCH", str(batch))
    _check(oracle, m, 400, 50, 1.0, 2)
