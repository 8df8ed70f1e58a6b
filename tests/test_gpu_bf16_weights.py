"""The window weights of the BF16 form's X, exact to FP32 rounding: one row of ones
in the first window and zeros elsewhere, so that X(r, j) = Upsilon(r, 0)
nu^(windows - 1). Bar: 1.3e-7, two roundings of 2^-24."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu,nwin", [(30.0, 8), (0.7, 70), (1.3, 100), (0.95, 300)])
def test_weight_of_the_first_window(lib_built, nu, nwin):
    import torch

    import skema_b200 as sk

    W, n = 64, 256
    A = torch.zeros(W * nwin, n, device="cuda")
    A[0] = 1.0
    with sk.SketchySVD(sk.AlgParams(matrix_m=W * nwin, matrix_n=n, rank=5, window=W, sketch_nu=nu,
                                    precision=sk._lib.PREC_BF16)) as s:
        U = s.map_export(sk._lib.UPSILON)[0][:, 0]
        s.linear_update(A)
        X = np.asarray(s.get_sketch(sk._lib.SKETCH_X), np.float64)
    want = U * float(np.float32(nu)) ** (nwin - 1)
    assert np.abs(X / want[:, None] - 1.0).max() < 1.3e-7
