"""CSR x SparseSign for few rows (four lanes per row) against the FP64 oracle,
around its tiles of eight rows, the runs of a row's four lanes and the row count
from which a lane takes a row alone. Bar: 1e-6, a row's few hundred terms."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,rank,nu", [(1, 30, 1, 1.0), (7, 50, 3, 1.0), (9, 400, 20, 0.5), (641, 700, 50, 0.9),
                                         (3000, 900, 60, 1.0), (14208, 300, 20, 1.0), (14217, 300, 20, 0.9)])
def test_against_the_oracle(lib_built, oracle, m, n, rank, nu):
    import torch

    import skema_b200 as sk

    rng = np.random.default_rng(m)
    cnt = rng.integers(0, 12, size=m)  # rows of 0 to 11 entries, one of many
    cnt[m // 2] = n // 2
    row = np.repeat(np.arange(m), cnt)
    A = sp.csr_matrix((rng.normal(size=row.size), (row, rng.integers(0, n, row.size))), shape=(m, n))
    A.sum_duplicates()
    A.data = A.data.astype(np.float32).astype(np.float64)
    w = max(1, m // 3)
    a = sk.AlgParams(matrix_m=m, matrix_n=n, rank=rank, window=w, sketch_nu=nu, issparse=True, dim_redux=1)
    o = oracle.OracleSketch(m, n, rank, w, kind=1, issparse=True, nu=nu)
    o.reset()
    rp = torch.from_numpy(A.indptr.astype(np.int64)).cuda()
    col, val = torch.from_numpy(A.indices).cuda(), torch.from_numpy(A.data.astype(np.float32)).cuda()
    with sk.SketchySVD(a) as s:
        s.reset()
        for r0, k in ((0, m - m // 4), (m - m // 4, m // 4)):
            s.update_rows((rp[r0:r0 + k + 1], col, val), r0)
            o.update_rows(A, r0, k)
        for name, g, want in zip("XYZ", s.get_sketches(), (o.X, o.Y, o.Z)):
            assert rel_fro(g, want) < 1e-6, name
