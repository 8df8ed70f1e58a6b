"""The FP32 sketch on the tensor cores (three BF16 planes per operand) against
the FP64 oracle, at the edges of its tiles and blocks.

Bar: 2e-6 relative Frobenius. Each operand is exact to 2^-24, a product drops
terms below 2^-24, a 32-deep run adds up to twelve FP32 terms without
round-to-nearest and the runs are added in FP32; with random signs these stay
well under 16 x 2^-24 = 1e-6 of the result's norm, twice that is the bar.
"""
import numpy as np
import pytest

from conftest import rel_fro

pytestmark = pytest.mark.gpu

BAR = 2e-6


@pytest.fixture(scope="module")
def sk(lib_built):
    import skema_b200

    return skema_b200


def _mat(m, n, seed):
    rng = np.random.default_rng(seed)
    p = min(m, n, 24)
    return ((rng.normal(size=(m, p)) * 10.0 ** (-0.2 * np.arange(p))) @ rng.normal(size=(p, n))
            + 1e-3 * rng.normal(size=(m, n))).astype(np.float32)


def _run(sk, oracle, A, rank, window, nu=1.0, inp=None, blocks=None, limit=0, **kw):
    m, n = A.shape
    a = sk.AlgParams(matrix_m=m, matrix_n=n, rank=rank, window=window, sketch_nu=nu, **kw)
    spd = bool(kw.get("issymmetric", False))
    o = oracle.OracleSketch(m, n, rank, window, nu=nu, spd=spd)
    with (sk.SketchySPD if spd else sk.SketchySVD)(a) as s:
        assert s.lib.skema_set_workspace_limit(s.h, limit) == 0
        o.reset()
        s.reset()
        for r0, w in blocks or [(0, m)]:
            s.update_rows((A if inp is None else inp)[r0:r0 + w], r0)
            o.update_rows(np.asarray(A, np.float64), r0, w)
        if spd:
            return [(s.get_sketches(), o.Y)]
        return list(zip(s.get_sketches(), (o.X, o.Y, o.Z)))


def _check(pairs):
    for q, (got, want) in enumerate(pairs):
        assert rel_fro(got, want) < BAR, (q, rel_fro(got, want))


@pytest.mark.parametrize("m,n,rank,window,order,nu", [
    (1000, 333, 5, 1000, "F", 1.0),    # one window, N tile of 64
    (3001, 1003, 10, 500, "C", 0.9),   # windows of unequal weight in one block
    (257, 2049, 16, 100, "F", 1.0),    # one row and one column past a tile
    (321, 4127, 30, 321, "C", 0.5),    # k = 121, s = 243
    (2048, 4096, 50, 1024, "F", 1.0),  # whole tiles, three N tiles
    (130, 9001, 3, 7, "C", 1.0),       # long rows, many short windows, k = 13
])
def test_dense_edges(sk, oracle, m, n, rank, window, order, nu):
    import torch

    A = _mat(m, n, m + n)
    t = torch.from_numpy(A).cuda()
    t = t if order == "C" else t.t().contiguous().t()
    _check(_run(sk, oracle, A, rank, window, nu, t))


@pytest.mark.parametrize("order", ["F", "C"])
def test_dense_unaligned_blocks_of_rows(sk, oracle, order):
    """Views off the 16-byte grid, a leading dimension that is no multiple of
    four, and blocks that start inside an 8-row group."""
    import torch

    big = torch.from_numpy(_mat(2003, 1501, 7)).cuda()
    big = big if order == "C" else big.t().contiguous().t()
    t = big[1:, 1:]
    _check(_run(sk, oracle, t.cpu().numpy(), 8, 300, 0.95, t, [(0, 701), (701, 1), (702, 1300)]))


def test_dense_row_blocks_under_a_workspace_limit(sk, oracle):
    """180 MB of planes within 200 MB: the call goes in several blocks."""
    import torch

    A = _mat(6000, 5000, 3)
    _check(_run(sk, oracle, A, 5, 900, 0.9, torch.from_numpy(A).cuda(), limit=200 << 20))


def test_spd(sk, oracle):
    import torch

    A = _mat(900, 900, 5)
    A = A + A.T
    _check(_run(sk, oracle, A, 12, 400, 1.0, torch.from_numpy(A).cuda(), issymmetric=True))


@pytest.mark.parametrize("N,d,window,order", [(700, 7, 300, "C"), (1300, 33, 1300, "F"), (901, 100, 128, "C")])
def test_rbf(sk, oracle, N, d, window, order):
    import torch

    P = oracle.mixture_points(N, d, seed=N)
    gamma = oracle.median_gamma(P)
    a = sk.AlgParams(matrix_m=N, matrix_n=N, rank=10, window=window, kernel_func=1, kernel_gamma=gamma,
                     force_three_sketch=True)
    o = oracle.OracleSketch(N, N, 10, window, kernel_gamma=gamma)
    o.linear_update(P)
    t = torch.from_numpy(P).cuda()
    with sk.SketchySVD(a) as s:
        s.linear_update(t if order == "C" else t.t().contiguous().t())
        _check(zip(s.get_sketches(), (o.X, o.Y, o.Z)))


@pytest.mark.parametrize("value", [2.0**101, np.inf, np.nan, -3.0e38])
def test_values_outside_the_planes_range(sk, value):
    """A value that the planes cannot carry gives what FP32 arithmetic gives:
    the same infinities and NaN, the other entries to the bar."""
    import torch

    m, n = 900, 800
    A = _mat(m, n, 1)
    A[123, 45] = value
    a = sk.AlgParams(matrix_m=m, matrix_n=n, rank=6, window=250)
    with sk.SketchySVD(a) as s:
        U, O, F, P = (s.map_export(w)[0].astype(np.float32) for w in range(4))
        s.linear_update(torch.from_numpy(A).cuda())
        X, Y, Z = s.get_sketches()
    with np.errstate(all="ignore"):
        big = abs(value) > 1e38  # products overflow FP32: only the pattern elsewhere is defined
        T = A.astype(np.float64) @ P.T.astype(np.float64)
        want = (U.astype(np.float64) @ A, A.astype(np.float64) @ O.T.astype(np.float64), F.astype(np.float64) @ T)
    for q, (g, w) in enumerate(zip((X, Y, Z), want)):
        fine = np.isfinite(w) & (np.abs(w) < 1e38)
        if not big or not np.isfinite(value):
            assert np.array_equal(np.isnan(g), np.isnan(w)), q
            assert np.array_equal(np.isposinf(g), np.isposinf(w)) and np.array_equal(np.isneginf(g), np.isneginf(w)), q
        hit = np.zeros_like(fine)
        if q == 0:
            hit[:, 45] = True
        elif q == 1:
            hit[123] = True
        else:
            hit[:] = True
        for part in (fine & ~hit, fine & hit):
            if part.any() and (not big or part is not None and not (part & hit).any()):
                assert rel_fro(g[part], w[part]) < 1e-5, q


def _pair64(P, gamma, Om, Yb):
    """Y = K Omega^T and the adjoint in FP64 by explicit differences."""
    P, Om, Yb = (np.asarray(t, np.float64) for t in (P, Om, Yb))
    d2 = np.maximum(((P[:, None, :] - P[None]) ** 2).sum(-1), 0.0)
    K = np.exp(-gamma * d2)
    np.fill_diagonal(K, 1.0)
    E = (Yb @ Om) * K
    np.fill_diagonal(E, 0.0)
    S = E + E.T
    return K @ Om.T, -2.0 * gamma * (S.sum(1)[:, None] * P - S @ P), -(E * d2).sum(), (np.abs(E) * d2).sum()


@pytest.mark.parametrize("N,d,k", [(1999, 3, 20), (1024, 24, 65), (1500, 70, 190), (1337, 129, 257)])
def test_pair(sk, oracle, N, d, k):
    """Forward and adjoint of the kernel sketch; dgamma is held against the sum
    of its terms' magnitudes, which it is a small difference of. Bar: 4e-6, the
    sketch's plus the FP32 distances and exponentials (a few 2^-24 of gamma d^2,
    of order one)."""
    import torch

    P = oracle.mixture_points(N, d, seed=N)
    gamma = oracle.median_gamma(P)
    rng = np.random.default_rng(N)
    Om, Yb = rng.normal(size=(k, N)).astype(np.float32), rng.normal(size=(N, k)).astype(np.float32)
    Yw, Xw, gw, gabs = _pair64(P, gamma, Om, Yb)
    t = [torch.from_numpy(a).cuda() for a in (P, Om, Yb)]
    Y = sk.rbf_sketch_fwd(t[0], gamma, t[1])
    dX, dg = sk.rbf_sketch_vjp(t[0], gamma, t[1], t[2])
    assert rel_fro(Y.cpu().numpy(), Yw) < 4e-6
    assert rel_fro(dX.cpu().numpy(), Xw) < 4e-6
    assert abs(dg - gw) < 4e-6 * gabs


@pytest.mark.parametrize("where,value", [("Om", np.inf), ("Yb", 2.0**105), ("Yb", np.nan), ("P", np.inf)])
def test_pair_values_outside_the_planes_range(sk, oracle, where, value):
    """What the SIMT form gives: the same calls under a workspace limit that
    leaves no room for the planes."""
    import torch

    from skema_b200.sketchy import _ctx_for_standalone

    N, d, k = 1600, 9, 70
    P = oracle.mixture_points(N, d, seed=2)
    gamma = oracle.median_gamma(P)
    rng = np.random.default_rng(5)
    a = {"P": P, "Om": rng.normal(size=(k, N)).astype(np.float32), "Yb": rng.normal(size=(N, k)).astype(np.float32)}
    a[where][3, 2] = value
    t = {q: torch.from_numpy(v).cuda() for q, v in a.items()}
    out = []
    for limit in (0, 32 << 20):
        with _ctx_for_standalone(0) as c:
            assert c.lib.skema_set_workspace_limit(c.h, limit) == 0
            Y = sk.rbf_sketch_fwd(t["P"], gamma, t["Om"], ctx=c).cpu().numpy()
            dX, dg = sk.rbf_sketch_vjp(t["P"], gamma, t["Om"], t["Yb"], ctx=c)
            out.append((Y, dX.cpu().numpy(), np.array([dg])))
    for g, w in zip(*out):
        assert np.array_equal(np.isnan(g), np.isnan(w)) and np.array_equal(np.isinf(g), np.isinf(w))
        f = np.isfinite(w)
        if f.any():
            assert rel_fro(g[f], w[f]) < 1e-5
