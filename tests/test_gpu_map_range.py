"""Imported Gauss maps whose values lie far from one, and sums that leave FP32's
range: the tensor-core FP32 form must give what FP32 arithmetic gives. Bars:
1e-5, the FP32 sketch's."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import rel_fro

pytestmark = pytest.mark.gpu

N, M, RANK, W = 300, 1300, 8, 65


def _input(form, A):
    import torch

    if form == "dense":
        return torch.from_numpy(A).cuda()
    B = sp.csr_matrix(A)
    return tuple(torch.from_numpy(q).cuda() for q in (B.indptr.astype(np.int64), B.indices.astype(np.int32), B.data))


def _run(form, A, scales, nu=1.0, positive=False, limit=0):
    """Device sketches and the FP64 ones for maps Upsilon, Omega, Phi, Psi scaled
    by 2^scales[i]."""
    import skema_b200 as sk

    a = sk.AlgParams(matrix_m=M, matrix_n=N, rank=RANK, window=W, sketch_nu=nu, issparse=form == "csr")
    with sk.SketchySVD(a) as s:
        assert s.lib.skema_set_workspace_limit(s.h, limit) == 0
        maps = []
        for i, e in enumerate(scales):
            v = s.map_export(i)[0] * 2.0**e
            v = np.abs(v) if positive else v
            s.map_import(i, v)
            maps.append(v if v.shape[1] in (M, N) else v.T)
        s.linear_update(_input(form, A))
        got = s.get_sketches()
    U, O, F, P = maps
    w = float(nu) ** ((M + W - 1) // W - 1 - np.arange(M) // W)
    with np.errstate(all="ignore"):
        A = A.astype(np.float64)
        return got, ((U * w) @ A, A @ O.T, (F * w) @ (A @ P.T))


@pytest.fixture(scope="module")
def A():
    rng = np.random.default_rng(1)
    a = rng.normal(size=(M, N)).astype(np.float32)
    a[rng.random(a.shape) < 0.8] = 0
    return a


@pytest.mark.parametrize("form", ["dense", "csr"])
@pytest.mark.parametrize("scales,nu,ascale", [
    ((95, 0, 95, 0), 4.0, -80),        # a weight of 4^19 on a map value of 2^95 is beyond FP32
    ((0, 0, 0, 0), 4.0, 0),
    ((-118, -118, -118, 0), 1.0, 0),   # maps that planes would carry with 16 bits
    ((0, -118, 0, -118), 1.0, 0),
    ((20, 20, 20, 20), 1.0, 20),
])
def test_finite(lib_built, form, scales, nu, ascale, A):
    got, want = _run(form, A * np.float32(2.0**ascale), scales, nu)
    for q, g, w in zip("XYZ", got, want):
        if form == "csr" and q in "XZ" and scales[0] == -118:
            continue  # FP32 atomics, which round values below 2^-126 to zero
        assert rel_fro(np.asarray(g, np.float64), w) < 1e-5, q


@pytest.mark.parametrize("form", ["dense", "csr"])
@pytest.mark.parametrize("scales,ascale", [((0, 0, 0, 70), 70), ((0, 0, 90, 30), 30), ((60, 60, 0, 0), 66)])
def test_overflow_is_an_infinity(lib_built, form, scales, ascale, A):
    """Sums of positive terms that pass FP32's largest value are +inf, not NaN."""
    got, want = _run(form, np.abs(A) * np.float32(2.0**ascale), scales, positive=True)
    for q, g, w in zip("XYZ", got, want):
        over, fine = w > 4e38, w < 3e38
        assert np.isposinf(g[over]).all(), q
        assert not np.isnan(g).any(), q
        if fine.any():
            assert rel_fro(np.asarray(g, np.float64)[fine], w[fine]) < 1e-5, q


@pytest.mark.parametrize("form", ["dense", "csr"])
@pytest.mark.parametrize("scales,ascale", [((-40, -40, -40, -40), 0), ((0, 0, 0, -30), -70), ((-49, -30, -20, -45), -60)])
def test_small_maps(lib_built, form, scales, ascale, A):
    """Maps that planes carry although their values are small, with A on either side
    of the bound that goes with Psi."""
    got, want = _run(form, A * np.float32(2.0**ascale), scales, 0.5)
    for q, g, w in zip("XYZ", got, want):
        if np.abs(w).max() > 2.0**-100:  # else FP32 atomics and accumulators round at 2^-149
            assert rel_fro(np.asarray(g, np.float64), w) < 1e-5, q
