"""Several windows of a call in one pass: their weights nu^(G-1-w), and the
BF16 form's X product over whole windows against one launch per window."""
import numpy as np
import pytest

from conftest import rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["dense", "csr"])
@pytest.mark.parametrize("nu,nwin,lo,hi", [
    (30.0, 40, 38, 40),  # nu^40 is beyond FP32, the data sit in the last windows
    (1e-3, 14, 0, 3),    # weights 1e-39 to 1e-33
    (0.0, 5, 0, 5),      # the last window alone counts
    (0.5, 90, 0, 90),    # two passes of 40 windows, one of 10
])
def test_weights_far_from_one(lib_built, oracle, form, nu, nwin, lo, hi):
    # Bar: 2e-6 as for one pass (each operand exact to 2^-24, terms below 2^-24
    # dropped), twice that for up to 14 roundings of nu X; 1e-5 for the CSR
    # form's X, whose sums have no fixed order.
    import scipy.sparse as sp
    import torch
    import skema_b200 as sk

    W, n = 64, 300
    m = nwin * W - 5
    rng = np.random.default_rng(nwin)
    A = rng.normal(size=(m, n)).astype(np.float32)
    A[: lo * W] = 0
    A[hi * W:] = 0
    if form == "csr":
        A[rng.random(A.shape) < 0.9] = 0
    B = sp.csr_matrix(A)
    o = oracle.OracleSketch(m, n, 10, W, nu=nu, issparse=form == "csr")
    o.reset()
    o.update_rows(B.astype(np.float64) if form == "csr" else A.astype(np.float64), 0, m)
    dev = [torch.from_numpy(q).cuda() for q in (B.indptr.astype(np.int64), B.indices.astype(np.int32), B.data)]
    with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=10, window=W, sketch_nu=nu,
                                    issparse=form == "csr")) as s:
        s.reset()
        s.update_rows(tuple(dev) if form == "csr" else torch.from_numpy(A).cuda(), 0)
        X, Y, Z = s.get_sketches()
    for got, want, bar in ((X, o.X, 1e-5 if form == "csr" else 4e-6), (Y, o.Y, 4e-6), (Z, o.Z, 4e-6)):
        assert rel_fro(np.asarray(got, np.float64), want) < bar


@pytest.mark.parametrize("m,n,order,window,nu", [
    (1000, 200, "F", 64, 0.9),     # 15 whole windows of one K step and a partial one
    (4133, 1132, "C", 512, 0.95),  # nine M tiles, the last of 108 columns
    (3072, 130, "F", 1024, 1.0),   # whole windows only, a last tile of two columns
    (640, 128, "C", 320, 0.5),
])
def test_bf16_windows_together(lib_built, m, n, order, window, nu):
    # The same BF16 operands and products; X's FP32 sums over at most 1024 rows
    # (64 tensor-core steps, each off by at most 2^-23 of the sum) are cut
    # differently: 64 x 2^-23 = 8e-6.
    import torch
    import skema_b200 as sk

    g = torch.Generator(device="cuda").manual_seed(m)
    buf = torch.randn(m * n + 4, device="cuda", generator=g)
    out = []
    for off in (0, 1):  # a base that TMA cannot address takes window after window
        v = torch.empty(m * n + 4, device="cuda")[off:off + m * n]
        v.copy_(buf[: m * n])
        A = v.view(n, m).t() if order == "F" else v.view(m, n)
        with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=10, window=window, sketch_nu=nu,
                                        precision=sk._lib.PREC_BF16)) as s:
            s.reset()
            s.update_rows(A, 0)
            s.update_rows(A, 0)  # X not empty
            out.append([np.array(q, np.float64) for q in s.get_sketches()])
    for a, b in zip(*out):
        assert rel_fro(a, b) < 8e-6
