"""FP32 sketches of values near the bottom of FP32's range, where the low BF16
planes of the tensor-core form run out of bits: the relative error stays what it
is at ordinary magnitudes (bars as in test_gpu_x3.py: 2e-6, 4e-6 for the kernel
pair). Scales are powers of two, so the inputs keep their bits: 2^-89 is carried
by the planes, 2^-95 and 2^-118 are not."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import rel_fro

pytestmark = pytest.mark.gpu

SCALES = [2.0**-89, 2.0**-95, 2.0**-118]


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("order,nu", [("F", 1.0), ("C", 0.9)])
def test_dense(lib_built, oracle, order, nu, scale):
    import torch

    import skema_b200 as sk

    m, n, rank, w = 900, 700, 8, 250
    A = np.random.default_rng(1).normal(size=(m, n)).astype(np.float32)
    o = oracle.OracleSketch(m, n, rank, w, nu=nu)
    o.linear_update(A.astype(np.float64))
    t = torch.from_numpy(A).cuda() * scale
    with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=rank, window=w, sketch_nu=nu)) as s:
        s.linear_update(t if order == "C" else t.t().contiguous().t())
        for q, g, want in zip("XYZ", s.get_sketches(), (o.X, o.Y, o.Z)):
            assert rel_fro(np.asarray(g, np.float64) / scale, want) < 2e-6, q


def test_small_entries_beside_ordinary_ones(lib_built, oracle):
    """What the planes lose of entries at 2^-118 is far below the others."""
    import torch

    import skema_b200 as sk

    m, n = 900, 700
    A = np.random.default_rng(2).normal(size=(m, n)).astype(np.float32)
    A[:, ::2] *= np.float32(2.0**-118)
    A[7] = 0
    o = oracle.OracleSketch(m, n, 8, m)
    o.linear_update(A.astype(np.float64))
    with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=8, window=m)) as s:
        s.linear_update(torch.from_numpy(A).cuda())
        for g, want in zip(s.get_sketches(), (o.X, o.Y, o.Z)):
            assert rel_fro(g, want) < 2e-6


@pytest.mark.parametrize("scale", SCALES)
def test_csr_gauss(lib_built, oracle, scale):
    """Y and Z; X is summed by FP32 atomics, which round values below 2^-126 to
    zero, in planes or not."""
    import torch

    import skema_b200 as sk

    m, n, w = 1100, 400, 300
    A = sp.random(m, n, density=0.05, format="csr", random_state=3, data_rvs=np.random.default_rng(3).standard_normal)
    A.data = A.data.astype(np.float32).astype(np.float64)
    o = oracle.OracleSketch(m, n, 9, w, issparse=True, nu=0.9)
    o.linear_update(A)
    t = (torch.from_numpy(A.indptr.astype(np.int64)).cuda(), torch.from_numpy(A.indices.astype(np.int32)).cuda(),
         torch.from_numpy(A.data.astype(np.float32)).cuda() * scale)
    with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=9, window=w, issparse=True, sketch_nu=0.9)) as s:
        s.linear_update(t)
        for q, g, want in zip("YZ", s.get_sketches()[1:], (o.Y, o.Z)):
            assert rel_fro(np.asarray(g, np.float64) / scale, want) < 2e-6, q


@pytest.mark.parametrize("scale", SCALES)
def test_pair(lib_built, oracle, scale):
    import torch

    import skema_b200 as sk
    from test_gpu_x3 import _pair64

    N, d, k = 1400, 6, 120
    P = oracle.mixture_points(N, d, seed=4)
    gamma = oracle.median_gamma(P)
    rng = np.random.default_rng(4)
    Om, Yb = rng.normal(size=(k, N)).astype(np.float32), rng.normal(size=(N, k)).astype(np.float32)
    Yw, Xw, gw, gabs = _pair64(P, gamma, Om, Yb)
    P, Om, Yb = (torch.from_numpy(a).cuda() for a in (P, Om, Yb))
    Y = sk.rbf_sketch_fwd(P, gamma, Om * scale)
    dX, dg = sk.rbf_sketch_vjp(P, gamma, Om, Yb * scale)
    assert rel_fro(Y.cpu().double().numpy() / scale, Yw) < 4e-6
    assert rel_fro(dX.cpu().double().numpy() / scale, Xw) < 4e-6
    assert abs(dg / scale - gw) < 4e-6 * gabs


@pytest.mark.parametrize("where", [slice(0, 7040), slice(7040, None), slice(0, 0)])
def test_adjoint_in_two_blocks(lib_built, oracle, where):
    """14,000 points take two blocks of rows; one, the other or none of them is
    too small for the planes."""
    import torch

    import skema_b200 as sk

    N, d, k = 14000, 3, 8
    P = oracle.mixture_points(N, d, seed=5)
    gamma = oracle.median_gamma(P)
    rng = np.random.default_rng(6)
    Om, Yb = rng.normal(size=(k, N)).astype(np.float32), rng.normal(size=(N, k)).astype(np.float32)
    Yb[where] *= np.float32(2.0**-118)
    P, Om, Yb = (torch.from_numpy(a).cuda() for a in (P, Om, Yb))
    dX, dg = sk.rbf_sketch_vjp(P, gamma, Om, Yb)
    x = P.double()
    d2 = torch.cdist(x, x, compute_mode="donot_use_mm_for_euclid_dist").square_()
    E = (Yb.double() @ Om.double()).mul_((d2 * -gamma).exp_())
    E.fill_diagonal_(0.0)
    want = -2.0 * gamma * ((E.sum(1) + E.sum(0))[:, None] * x - E @ x - E.t() @ x)
    assert rel_fro(dX.cpu().numpy(), want.cpu().numpy()) < 4e-6
    E.mul_(d2)
    assert abs(dg + float(E.sum())) < 4e-6 * float(E.abs().sum())
