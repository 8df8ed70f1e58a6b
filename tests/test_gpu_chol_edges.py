"""Cholesky, triangular inverse and solve of the approximation at the edges of
their 8-wide blocks and of the shared-memory form (k up to 225 and past it):
the approximation of the device's own sketches against the oracle's, which
takes LAPACK's QR, solves and SVD. Bar: the approximation tests' 1e-9 of the
largest singular value."""
import numpy as np
import pytest

from conftest import rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 31, 64, 113, 114, 115, 129, 200, 224, 225, 226, 256, 257])
def test_approximation(lib_built, oracle, k):
    import skema_b200 as sk

    m, n, r, s = 700, 610, min(k, 5), 2 * k + 1
    rng = np.random.default_rng(k)
    p = 40
    A = ((rng.normal(size=(m, p)) * 10.0 ** (-0.1 * np.arange(p))) @ rng.normal(size=(p, n))
         + 0.01 * rng.normal(size=(m, n))).astype(np.float32)
    a = sk.AlgParams(matrix_m=m, matrix_n=n, rank=r, window=m, sketch_range=k, sketch_core=s)
    o = oracle.OracleSketch(m, n, r, m, sketch_range=k, sketch_core=s)
    with sk.SketchySVD(a) as c:
        c.linear_update(A)
        X, Y, Z = (np.asarray(t, np.float64) for t in c.get_sketches())
        for which, key in ((0, "upsilon"), (1, "omega"), (2, "phi"), (3, "psi")):
            o.maps[key]._dense = c.map_export(which)[0]
        U, S, V = c.low_rank_approx()
    o.X, o.Y, o.Z = X, Y, Z
    Uo, So, Vo = o.low_rank_approx()
    assert np.abs(S - So).max() < 1e-9 * So[0]
    assert rel_fro((U * S) @ V.T, (Uo * So) @ Vo.T) < 1e-8
