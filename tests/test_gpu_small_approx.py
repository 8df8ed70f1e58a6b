"""The approximation of small sketches: ranges around the one up to which the
Cholesky kernel forms the inverse itself (32) and the one from which Gram matrices
of fewer than 1,024 rows are plain products (40), with few rows; rank-deficient
sketches at every form of the core SVD. Bar: 1e-9 of the largest singular value,
as test_gpu_chol_edges.py."""
import numpy as np
import pytest

from conftest import rel_fro

pytestmark = pytest.mark.gpu


def _check(oracle, m, n, k, p, noise):
    import skema_b200 as sk

    r, s = min(k, 5, p), 2 * k + 1
    rng = np.random.default_rng(k + m)
    A = ((rng.normal(size=(m, p)) * 10.0 ** (-0.1 * np.arange(p))) @ rng.normal(size=(p, n))
         + noise * rng.normal(size=(m, n))).astype(np.float32)
    a = sk.AlgParams(matrix_m=m, matrix_n=n, rank=r, window=m, sketch_range=k, sketch_core=s)
    o = oracle.OracleSketch(m, n, r, m, sketch_range=k, sketch_core=s)
    with sk.SketchySVD(a) as c:
        c.linear_update(A)
        X, Y, Z = (np.asarray(t, np.float64) for t in c.get_sketches())
        for which, key in ((0, "upsilon"), (1, "omega"), (2, "phi"), (3, "psi")):
            o.maps[key]._dense = c.map_export(which)[0]
        U, S, V = c.low_rank_approx()
        sweeps = c.timing_get("approx.svd_sweeps")[1]
    o.X, o.Y, o.Z = X, Y, Z
    return A, (U, S, V), o.low_rank_approx(), sweeps


@pytest.mark.parametrize("k", [3, 15, 16, 17, 32, 33, 40, 41])
@pytest.mark.parametrize("m,n", [(63, 1023), (65, 1025), (1023, 64)])
def test_small(lib_built, oracle, m, n, k):
    _, (U, S, V), (Uo, So, Vo), _ = _check(oracle, m, n, k, 40, 0.01)
    assert np.abs(S - So).max() < 1e-9 * So[0]
    assert rel_fro((U * S) @ V.T, (Uo * So) @ Vo.T) < 1e-8


@pytest.mark.parametrize("k", [9, 41, 81, 113, 117, 161, 201, 225, 256])
@pytest.mark.parametrize("p", [1, 6])
def test_rank_deficient(lib_built, k, p, oracle):
    """A of rank p < k: the bases are completed from the Gram matrices' eigenvectors
    (jacobi_svd_kernel to k = 114, jacobi_cluster_kernel above), and the result is A
    to the rounding of its FP32 sketches (1e-5). The core SVD ends by itself, well
    before its limit of 60 sweeps."""
    A, (U, S, V), _, sweeps = _check(oracle, 700, 610, k, p, 0.0)
    A = A.astype(np.float64)
    r = len(S)
    Ua, Sa, Va = np.linalg.svd(A, full_matrices=False)
    best = (Ua[:, :r] * Sa[:r]) @ Va[:r]
    assert np.abs(U.T @ U - np.eye(r)).max() < 1e-9 and np.abs(V.T @ V - np.eye(r)).max() < 1e-9
    assert rel_fro((U * S) @ V.T, best) < 1e-5
    assert 0 < sweeps < 30, sweeps


@pytest.mark.parametrize("k", [9, 41, 81, 113, 117, 161, 201, 225, 256])
@pytest.mark.parametrize("p", [1, 6])
def test_exactly_rank_deficient_sketches(lib_built, k, p):
    """Sketches of an integer matrix of rank p whose Y and X are of rank p exactly
    (factors of few bits), so that no Cholesky factor exists and the eigenvectors
    of a Gram matrix with k - p zero eigenvalues are taken: U S V^T is the matrix
    to the rounding of Z (1e-5)."""
    import skema_b200 as sk
    from skema_b200 import _lib as L

    m, n, s, r = 700, 610, 2 * k + 1, min(p, 5)
    rng = np.random.default_rng(100 * k + p)
    a, b = rng.integers(-4, 5, size=(m, p)).astype(float), rng.integers(-4, 5, size=(n, p)).astype(float)
    al = sk.AlgParams(matrix_m=m, matrix_n=n, rank=r, window=m, sketch_range=k, sketch_core=s)
    with sk.SketchySVD(al) as c:
        O, F, P = (c.map_export(w)[0] for w in (L.OMEGA, L.PHI, L.PSI))
        U = c.map_export(L.UPSILON)[0]
        few = lambda t: np.round(t * 8) / 8  # |values| below 2^10: factors of 13 bits and 3
        Y, X = a @ few(b.T @ O.T), few(U @ a) @ b.T
        assert np.array_equal(Y, Y.astype(np.float32)) and np.array_equal(X, X.astype(np.float32))
        Z = (F @ a) @ (P @ b).T
        for which, t in ((L.SKETCH_X, X), (L.SKETCH_Y, Y), (L.SKETCH_Z, Z)):
            c.set_sketch(which, t.astype(np.float32))
        l0 = c.launch_count()
        Uo, So, Vo = c.low_rank_approx()
        launches = c.launch_count() - l0
        # the same call on sketches of full rank
        for which, t in ((L.SKETCH_X, X), (L.SKETCH_Y, Y), (L.SKETCH_Z, Z)):
            c.set_sketch(which, rng.normal(size=t.shape).astype(np.float32))
        l0 = c.launch_count()
        c.low_rank_approx()
        plain = c.launch_count() - l0
    A = a @ b.T
    Ua, Sa, Va = np.linalg.svd(A, full_matrices=False)
    best = (Ua[:, :r] * Sa[:r]) @ Va[:r]
    assert np.abs(Uo.T @ Uo - np.eye(r)).max() < 1e-9 and np.abs(Vo.T @ Vo - np.eye(r)).max() < 1e-9
    assert rel_fro((Uo * So) @ Vo.T, best) < 1e-5
    # a basis by way of the eigenvectors takes launches that a plain one does not;
    # how many depends on which Cholesky fails first, and so on rounding
    assert launches > plain, (launches, plain)
