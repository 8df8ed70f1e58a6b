"""CSR x Gauss on both sides of the row count (32 rows per SM) from which a CTA takes
32 rows instead of 8, rows added to a Y that is not empty among them. Bars as in
test_gpu_csr_gauss.py."""
import pytest

from conftest import rel_fro
from test_gpu_csr_gauss import _csr, _dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("past", [-1, 0, 33])
@pytest.mark.parametrize("spd", [False, True])
def test_at_the_line(lib_built, oracle, past, spd):
    import torch

    import skema_b200 as sk

    m = 32 * torch.cuda.get_device_properties(0).multi_processor_count + past
    A = _csr(m, m if spd else 700, 4, 5)
    a = sk.AlgParams(matrix_m=m, matrix_n=A.shape[1], rank=10, window=m // 3, sketch_nu=0.9, issparse=True, issymmetric=spd)
    o = oracle.OracleSketch(m, A.shape[1], 10, m // 3, issparse=True, nu=0.9, spd=spd)
    o.reset()
    with (sk.SketchySPD if spd else sk.SketchySVD)(a) as s:
        s.reset()
        for _ in range(2):
            s.update_rows(_dev(A), 0)
            o.update_rows(A, 0, m)
        got = s.get_sketches()
    if spd:
        assert rel_fro(got, o.Y) < 2e-6
        return
    for name, g, w, bar in zip("XYZ", got, (o.X, o.Y, o.Z), (1e-5, 2e-6, 2e-6)):
        assert rel_fro(g, w) < bar, (name, rel_fro(g, w))
