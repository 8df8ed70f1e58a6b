"""The residual pass's FP64 products at the edges of their tiles (column counts
around the multiples of eight, both storage orders, K splits) and over several
row blocks, against the oracle's restatement. Bar: the FP64 pass's 1e-9."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,r,window,order", [
    (300, 129, 1, 300, "F"), (1025, 300, 7, 400, "C"), (2100, 1030, 17, 2100, "F"), (1500, 2600, 33, 70, "C"),
    (1200, 515, 65, 1200, "F"), (70001, 65, 9, 70001, "C"),
])
def test_against_the_oracle(lib_built, oracle, m, n, r, window, order):
    import torch

    import skema_b200 as sk
    from oracle import sketchy_oracle

    rng = np.random.default_rng(m)
    A = rng.normal(size=(m, n)).astype(np.float32)
    U, V = rng.normal(size=(m, r)), rng.normal(size=(n, r))
    S = np.sort(rng.uniform(1, 9, r))[::-1].copy()
    t = torch.from_numpy(A).cuda()
    t = t if order == "C" else t.t().contiguous().t()
    with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=r, window=window, sketch_range=r, sketch_core=r)) as s:
        got = s.residuals(t, U, S, V)
    want = sketchy_oracle.residuals(A.astype(np.float64), U, S, V)
    assert np.allclose(got, want, rtol=1e-9, atol=0)
