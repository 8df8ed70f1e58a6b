"""Device fetches of the sketches in the layout they are not stored in: the
values are moved, so every layout and leading dimension gives the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 40, 3), (31, 33, 7), (64, 40, 8), (1000, 97, 81), (4097, 65, 256), (333, 70, 301)])
def test_layouts_agree(lib_built, m, n, k):
    import ctypes as C

    import torch

    import skema_b200 as sk
    from skema_b200 import _lib as L

    a = sk.AlgParams(matrix_m=m, matrix_n=n, rank=1, sketch_range=k, sketch_core=4)
    g = torch.Generator(device="cuda").manual_seed(k)
    with sk.SketchySVD(a) as s:
        for which, (r, c) in ((L.SKETCH_Y, (m, k)), (L.SKETCH_X, (k, n))):
            want = torch.randn(r, c, generator=g, device="cuda")
            s.set_sketch(which, want)
            for layout, extra, off in ((0, 0, 0), (1, 0, 0), (0, 5, 0), (1, 3, 0), (0, 0, 1), (1, 0, 1)):
                inner, outer = (r, c) if layout == 0 else (c, r)
                buf = torch.full((off + outer * (inner + extra),), 7.0, device="cuda")
                torch.cuda.synchronize()
                s._check(s.lib.skema_get_sketch(s.h, which, C.c_void_p(buf.data_ptr() + 4 * off), inner + extra, layout,
                                                L.MEM_DEVICE))
                s.synchronize()
                got = buf[off:].reshape(outer, inner + extra)
                assert torch.equal(got[:, :inner], want.t() if layout == 0 else want), (which, layout, extra, off)
                assert np.all(got[:, inner:].cpu().numpy() == 7.0) and (not off or float(buf[0]) == 7.0)
