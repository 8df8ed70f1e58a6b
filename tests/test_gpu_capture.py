"""FP32 updates under stream capture: a call of several windows is captured after a
warm-up of one window, so the workspace cannot grow; the graph's sketches are
those of the plain call (bar 1e-5, the two forms' rounding and sums in no fixed
order)."""
import pytest

from conftest import rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["dense", "rbf", "csr"])
def test_capture_after_a_smaller_warm_up(lib_built, form):
    import torch

    import skema_b200 as sk

    m, n, w = 3000, 3000, 300
    g = torch.Generator(device="cuda").manual_seed(1)
    kw = {}
    A = torch.randn(m, n, generator=g, device="cuda")
    if form == "rbf":
        A, kw = A[:, :9].contiguous(), dict(kernel_func=1, kernel_gamma=0.05, force_three_sketch=True)
    elif form == "csr":
        S = A.where(A > 1.5, 0).to_sparse_csr()
        A, kw = (S.crow_indices().long(), S.col_indices().int(), S.values()), dict(issparse=True)
    first = A if form == "rbf" else (A[0][: w + 1], A[1], A[2]) if form == "csr" else A[:w]
    out = []
    for captured in (False, True):
        with sk.SketchySVD(sk.AlgParams(matrix_m=m, matrix_n=n, rank=10, window=w, sketch_nu=0.9, **kw)) as s:
            res = [torch.zeros(q, device="cuda") for q in ((s.range, n), (m, s.range), (s.core, s.core))]

            def fetch():
                for q in range(3):
                    s.get_sketch(q, out=res[q])

            s.reset()
            s.update_rows(first, 0, w) if form == "rbf" else s.update_rows(first, 0)
            fetch()
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            if captured:
                with torch.cuda.graph(graph):
                    s.reset()
                    s.update_rows(A, 0)
                    fetch()
                for t in res:
                    t.zero_()
                graph.replay()
            else:
                s.reset()
                s.update_rows(A, 0)
                fetch()
            torch.cuda.synchronize()
            out.append([t.cpu().numpy() for t in res])
            del graph
    for q, a, b in zip("XYZ", *out):
        assert rel_fro(b, a) < 1e-5, q
