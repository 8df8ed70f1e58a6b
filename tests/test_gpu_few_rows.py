"""FP32 dense calls of few rows on a wide matrix (tensor-core products whose K is
one to four steps of 32, added to sketches that are not empty) against the FP64
oracle. Bar: test_gpu_x3.py's 2e-6."""
import numpy as np
import pytest

from conftest import rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rank,nu,rows", [
    (9000, 30, 1.0, (1, 32, 33, 64)),    # N tiles of 128 and 192 columns
    (9000, 30, 0.5, (65, 96, 97, 128)),
    (30001, 4, 1.0, (16, 15, 63, 129)),  # 235 M tiles of X, more than CTAs
])
def test_against_the_oracle(lib_built, oracle, n, rank, nu, rows):
    import torch

    import skema_b200 as sk

    m = sum(rows)
    A = np.random.default_rng(n).normal(size=(m, n)).astype(np.float32)
    o = oracle.OracleSketch(m, n, rank, 50, nu=nu)
    o.reset()
    t = torch.from_numpy(A).cuda()
    with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=rank, window=50, sketch_nu=nu)) as s:
        s.reset()
        r0 = 0
        for w in rows:
            s.update_rows(t[r0:r0 + w], r0)
            o.update_rows(A.astype(np.float64), r0, w)
            r0 += w
        for q, g, want in zip("XYZ", s.get_sketches(), (o.X, o.Y, o.Z)):
            assert rel_fro(g, want) < 2e-6, q
