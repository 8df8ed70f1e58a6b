"""Ordering against torch's streams: inputs still being written and outputs
still being read on torch's current stream, whichever that is."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own_stream", [False, True])
def test_inputs_and_outputs_are_ordered(lib_built, own_stream):
    import torch

    import skema_b200 as sk
    from skema_b200 import _lib as L

    m, n = 3000, 1200
    a = sk.AlgParams(matrix_m=m, matrix_n=n, rank=8, window=m)
    A = torch.randn(m, n, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    with sk.SketchySVD(a) as s:
        s.linear_update(A)
        want = s.get_sketch(L.SKETCH_Y, out=torch.empty(m, s.range, device="cuda"))
        torch.cuda.synchronize()
        st = torch.cuda.Stream() if own_stream else torch.cuda.current_stream()
        busy = torch.empty(64 << 20, device="cuda")
        with torch.cuda.stream(st):
            for _ in range(3):
                for _ in range(40):
                    busy.mul_(1.0)  # the input is written only after this
                B = torch.empty_like(A).copy_(A)
                out = torch.full((m, s.range), 3.0, device="cuda")
                s.linear_update(B)
                s.get_sketch(L.SKETCH_Y, out=out)
                B.zero_()  # after the library's reads of it
                del B
                assert torch.equal(out, want)  # torch reads after the library's write


def test_order_streams_status(lib_built):
    import skema_b200 as sk
    from skema_b200 import _lib as L

    with sk.SketchySVD(sk.AlgParams(matrix_m=4, matrix_n=4)) as s:
        assert s.lib.skema_order_streams(None, None, 1) == L.EINVAL
        assert s.lib.skema_order_streams(s.h, None, 1) == L.OK  # the legacy default stream
        assert s.lib.skema_order_streams(s.h, None, 0) == L.OK
