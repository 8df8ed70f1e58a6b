"""A fetch to device memory in an FP32 context does not wait on the host, with or
without the tensor-core form's update before it; the status word is read by the
next call that waits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["dense", "rbf", "csr"])
def test_update_and_fetch_return_while_the_stream_is_busy(lib_built, form):
    import torch

    import skema_b200 as sk
    from skema_b200 import _lib as L

    m, n = 2048, 2048
    g = torch.Generator(device="cuda").manual_seed(1)
    kw = {}
    A = torch.randn(m, n, generator=g, device="cuda")
    if form == "rbf":
        A, kw = A[:, :16].contiguous(), dict(kernel_func=1, kernel_gamma=0.03, force_three_sketch=True)
    elif form == "csr":
        S = A.where(A > 1.5, 0).to_sparse_csr()
        A, kw = (S.crow_indices().long(), S.col_indices().int(), S.values()), dict(issparse=True)
    with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=8, window=700, **kw)) as s:
        shapes = ((s.range, n), (m, s.range), (s.core, s.core))
        out = [torch.zeros(q, device="cuda") for q in shapes]

        def step():
            s.reset()
            s.update_rows(A, 0)
            for w in range(3):
                s.get_sketch(w, out=out[w])

        step()
        s.synchronize()
        want = [t.clone() for t in out]
        for t in out:
            t.zero_()
        torch.cuda.synchronize()
        torch.cuda._sleep(400_000_000)  # 0.2 s or more of the stream that the library waits for
        step()
        done = torch.cuda.Event()
        done.record()
        assert not done.query()
        s.synchronize()
        torch.cuda.synchronize()
        for q, a, b in zip("XYZ", out, want):
            assert torch.allclose(a, b, rtol=1e-4, atol=1e-4 * float(b.abs().max())), q


def test_time_out_is_reported_by_the_next_waiting_call(lib_built):
    import torch

    import skema_b200 as sk
    from skema_b200 import _lib as L

    m, n = 4096, 2048
    A = torch.randn(m, n, device="cuda")
    for fetch in ("synchronize", "host"):
        with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=8, window=1024)) as s:
            out = torch.empty(m, s.range, device="cuda")
            s.linear_update(A)
            want = s.get_sketch(L.SKETCH_Y)
            assert s.lib.skema_set_wait_limit(s.h, 1) == L.OK
            s.linear_update(A)
            s.get_sketch(L.SKETCH_Y, out=out)
            with pytest.raises(sk.SkemaError) as e:
                s.synchronize() if fetch == "synchronize" else s.get_sketch(L.SKETCH_Y)
            assert e.value.status == L.ETIMEOUT
            assert s.lib.skema_set_wait_limit(s.h, 0) == L.OK
            s.linear_update(A)
            assert np.array_equal(s.get_sketch(L.SKETCH_Y), want)
