"""The forms that FP32 updates take when the tensor-core ones are not to be had:
CSR x Gauss window by window under a workspace limit, imported maps with huge
values, and the products of blocks with infinities against the SIMT windows."""
import numpy as np
import pytest

from conftest import rel_fro
from test_gpu_csr_gauss import _csr, _dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu", [1.0, 0.9])
def test_csr_gauss_under_a_workspace_limit(lib_built, oracle, nu):
    """8 MB hold the n x s scratch of a window, not the one-pass form's 39 MB of parts.
    Bar: 1e-5, FP32 sums in no fixed order."""
    import skema_b200 as sk

    m, n, rank, w = 3000, 800, 15, 700
    A = _csr(m, n, 9, 11)
    o = oracle.OracleSketch(m, n, rank, w, issparse=True, nu=nu)
    o.reset()
    rp, col, val = _dev(A)
    with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=rank, window=w, sketch_nu=nu, issparse=True)) as s:
        assert s.lib.skema_set_workspace_limit(s.h, 8 << 20) == 0
        s.reset()
        for r0, k in ((0, 1601), (1601, 1399), (0, 1000)):
            s.update_rows((rp[r0:r0 + k + 1], col, val), r0)
            o.update_rows(A, r0, k)
        for q, g, want in zip("XYZ", s.get_sketches(), (o.X, o.Y, o.Z)):
            assert rel_fro(g, want) < 1e-5, q


@pytest.mark.parametrize("form", ["dense", "csr", "rbf"])
@pytest.mark.parametrize("which", [0, 1, 2, 3])
def test_one_huge_map_value(lib_built, oracle, form, which):
    """An imported map with one value of 2^101: the sketch that it enters holds it to
    FP32 rounding, the others are as without it. Bar: 1e-5."""
    import torch

    import skema_b200 as sk

    m, n, rank = 900, 900, 8
    P = oracle.mixture_points(m, 5, seed=1)
    gamma = oracle.median_gamma(P)
    kw = dict(kernel_func=1, kernel_gamma=gamma, force_three_sketch=True) if form == "rbf" else dict(issparse=form == "csr")
    if form == "rbf":
        D = np.exp(-gamma * ((P.astype(np.float64)[:, None] - P.astype(np.float64)[None]) ** 2).sum(-1))
        t = torch.from_numpy(P).cuda()
    else:
        B = _csr(m, n, 20, 2)
        D, t = B.toarray(), _dev(B) if form == "csr" else torch.from_numpy(B.toarray().astype(np.float32)).cuda()
    with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=rank, window=300, **kw)) as s:
        maps = [s.map_export(i)[0] for i in range(4)]
        maps[which][5, 3] = 2.0**101
        s.map_import(which, maps[which])
        s.linear_update(t)
        got = s.get_sketches()
    U, O, F, Q = (v if v.shape[1] == n else v.T for v in maps)
    for q, g, want in zip("XYZ", got, (U @ D, D @ O.T, F @ (D @ Q.T))):
        assert rel_fro(np.asarray(g, np.float64), want) < 1e-5, q


@pytest.mark.parametrize("order", ["F", "C"])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, -3.0e38, 2.0**101])
def test_non_finite_patterns(lib_built, order, value):
    """One call (products of a refused block) and calls of 150 rows, which are too
    small for the tensor-core form: the same infinities, NaN and finite values."""
    import torch

    import skema_b200 as sk

    m, n = 900, 800
    rng = np.random.default_rng(3)
    A = rng.normal(size=(m, n)).astype(np.float32)
    A[123, 45] = value
    t = torch.from_numpy(A).cuda()
    t = t if order == "C" else t.t().contiguous().t()
    out = []
    for step in (m, 150):
        with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=6, window=m)) as s:
            s.reset()
            for r in range(0, m, step):
                s.update_rows(t[r:r + step], r)
            out.append([np.asarray(q, np.float64) for q in s.get_sketches()])
    for q, a, b in zip("XYZ", *out):
        assert np.array_equal(np.isnan(a), np.isnan(b)), q
        assert np.array_equal(np.isposinf(a), np.isposinf(b)) and np.array_equal(np.isneginf(a), np.isneginf(b)), q
        f = np.isfinite(b)
        if f.any():
            assert rel_fro(a[f], b[f]) < 1e-5, q
