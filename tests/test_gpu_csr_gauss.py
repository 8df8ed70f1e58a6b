"""CSR input with Gauss maps against the FP64 oracle, at the edges of the
gather kernel's tiles and of the row blocks. Bar: the FP32 sketch's 1e-5 for
sums in no fixed order (X), 2e-6 elsewhere (a row's few dozen terms; Z through
the three-plane product)."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import rel_fro

pytestmark = pytest.mark.gpu


def _csr(m, n, mean, seed):
    """Rows of 0 to many entries, one of them half full; sorted columns."""
    rng = np.random.default_rng(seed)
    cnt = np.minimum((mean / 1.65 * np.exp(rng.normal(size=m))).astype(np.int64), n)
    cnt[:: max(m // 7, 1)] = 0
    cnt[m // 2] = max(n // 2, 1)
    row = np.repeat(np.arange(m), cnt)
    A = sp.csr_matrix((rng.normal(size=row.size), (row, rng.integers(0, n, row.size))), shape=(m, n))
    A.sum_duplicates()
    A.data = A.data.astype(np.float32).astype(np.float64)
    return A


def _dev(A):
    import torch

    return (torch.from_numpy(A.indptr.astype(np.int64)).cuda(), torch.from_numpy(A.indices.astype(np.int32)).cuda(),
            torch.from_numpy(A.data.astype(np.float32)).cuda())


def _compare(sk, oracle, A, rank, window, nu=1.0, blocks=None, spd=False, **kw):
    m, n = A.shape
    a = sk.AlgParams(matrix_m=m, matrix_n=n, rank=rank, window=window, sketch_nu=nu, issparse=True, issymmetric=spd, **kw)
    o = oracle.OracleSketch(m, n, rank, window, issparse=True, nu=nu, spd=spd, **kw)
    rp, col, val = _dev(A)
    with (sk.SketchySPD if spd else sk.SketchySVD)(a) as s:
        s.reset()
        for r0, w in blocks or [(0, m)]:
            s.update_rows((rp[r0:r0 + w + 1], col, val), r0)
            o.update_rows(A, r0, w)
        got = s.get_sketches()
    if spd:
        assert rel_fro(got, o.Y) < 2e-6
        return
    for name, g, w, bar in zip("XYZ", got, (o.X, o.Y, o.Z), (1e-5, 2e-6, 2e-6)):
        assert rel_fro(g, w) < bar, (name, rel_fro(g, w))


@pytest.mark.parametrize("m,n,rank,window,nu,blocks", [
    (33, 20, 2, 33, 1.0, None),                             # a tile and one row
    (1000, 300, 15, 130, 0.9, None),                        # k + s = 184, several weighted windows
    (777, 500, 70, 200, 1.0, [(0, 100), (100, 1), (101, 676)]),  # k + s = 844: four column passes
    (2500, 4000, 21, 2500, 0.5, [(0, 1700), (1700, 800)]),  # k = 85: a partial group of four
])
def test_edges(lib_built, oracle, m, n, rank, window, nu, blocks):
    import skema_b200 as sk

    _compare(sk, oracle, _csr(m, n, 9, m), rank, window, nu, blocks)


def test_two_row_blocks(lib_built, oracle):
    import skema_b200 as sk

    _compare(sk, oracle, _csr(17000, 60, 5, 4), 3, 4000, 0.9, sketch_range=13, sketch_core=2000)


def test_spd(lib_built, oracle):
    import skema_b200 as sk

    A = _csr(400, 400, 9, 3)
    _compare(sk, oracle, (A + A.T).tocsr(), 20, 130, spd=True)


@pytest.mark.parametrize("value", [2.0**104, np.inf, np.nan])
def test_values_outside_the_planes_range(lib_built, value):
    """The Z product falls back to FP32 arithmetic: its infinities and NaN."""
    import skema_b200 as sk

    A = _csr(600, 200, 9, 8)
    A.data[A.indptr[77]] = value
    a = sk.AlgParams(matrix_m=600, matrix_n=200, rank=5, window=250, issparse=True)
    with sk.SketchySVD(a) as s:
        M = [s.map_export(w)[0] for w in range(4)]
        s.linear_update(_dev(A))
        X, Y, Z = s.get_sketches()
    D = A.toarray()
    mask = D == 0  # an absent entry adds nothing, also beside an infinity
    T = np.array([sum((D[i, j] * M[3][j] for j in np.flatnonzero(~mask[i])), np.zeros(M[3].shape[1])) for i in range(600)])
    with np.errstate(all="ignore"):
        want = M[2].T @ T
    assert np.array_equal(np.isnan(Z), np.isnan(want))
    assert np.array_equal(np.isinf(Z), np.isinf(want))
    f = np.isfinite(want)
    if f.any():
        assert rel_fro(Z[f], want[f]) < 1e-5
