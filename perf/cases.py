"""The workloads by which this library's speed is judged.

Each case is one pass through the public Python API on device data, as a
streaming SketchySVD program runs it: a sketch update over all rows with the
three sketches read back into the program's own buffers, the kernel-sketch
forward and adjoint, or the fixed-rank approximation followed by its residual
pass. Sizes are those of the benchmark's configurations, smaller and ragged
ones of the same recipes, and draws over the same ranges. `exact` restates the
result in FP64 with plain torch, maps included.
"""
from __future__ import annotations

import math

import torch

import skema_b200 as sk
from skema_b200 import _lib as L

DEV = "cuda"


# ------------------------------------------------------------------ cases --
def _csr(m, n, nnz_row, rows, maps, rank, window, nu=1.0):
    return dict(kind="csr", m=m, n=n, nnz_row=nnz_row, rows=rows, maps=maps, rank=rank, window=window, nu=nu)


def _dense(m, n, layout, maps, precision, rank, window, nu=1.0):
    return dict(kind="dense", m=m, n=n, layout=layout, maps=maps, precision=precision, rank=rank, window=window, nu=nu)


def _rbf(m, d, precision, rank, window):
    return dict(kind="rbf", m=m, d=d, precision=precision, rank=rank, window=window)


def _pair(m, d, k, precision):
    return dict(kind="pair", m=m, d=d, k=k, precision=precision)


def _approx(m, n, source, rank, window):
    return dict(kind="approx", m=m, n=n, source=source, rank=rank, window=window)


def listed():
    return [
        # The smallest call: one short block of sparse rows, as a program that
        # sketches a stream as it arrives sends it. Launches and host time.
        dict(_csr(2000, 500, 10, "skewed", "sign", 10, 2000), name="csr-sign-small"),
        # The benchmark's default: a million sparse rows, sparse-sign maps.
        dict(_csr(1_000_000, 100_000, 10, "even", "sign", 20, 10_000), name="csr-sign-1m"),
        # Sparse input with the default (Gauss) maps, uneven row lengths.
        dict(_csr(100_000, 20_000, 10, "skewed", "gauss", 20, 10_000), name="csr-gauss"),
        # A small dense matrix in row-major order, odd sizes, several windows.
        dict(_dense(3001, 1003, "row", "gauss", "fp32", 10, 500), name="dense-fp32-small"),
        # A quarter of the rows of the benchmark's dense case, default precision.
        dict(_dense(50_000, 20_000, "col", "gauss", "fp32", 50, 8192), name="dense-fp32"),
        # The benchmark's dense case in the tensor-core form.
        dict(_dense(200_000, 20_000, "col", "gauss", "bf16", 50, 8192), name="dense-bf16"),
        # Gauss-RBF kernel input, default precision, a feature count that is
        # no multiple of a tile.
        dict(_rbf(40_000, 100, "fp32", 32, 4096), name="rbf-fp32"),
        # The benchmark's kernel case: 100,000 points in 128 dimensions.
        dict(_rbf(100_000, 128, "bf16", 64, 4096), name="rbf-bf16"),
        # Kernel sketch and its gradient (points and gamma): a training step.
        dict(_pair(20_000, 24, 65, "fp32"), name="pair-fp32"),
        dict(_pair(50_000, 64, 129, "bf16"), name="pair-bf16"),
        # Fixed-rank approximation and residual norms after the update: the
        # sketches of the default sparse benchmark, and a dense matrix of
        # decaying spectrum.
        dict(_approx(1_000_000, 100_000, "csr", 20, 10_000), name="approx-csr"),
        dict(_approx(50_000, 10_000, "dense", 50, 8192), name="approx-dense"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["csr", "csr", "dense", "dense", "rbf", "pair", "approx"])
    nu = rng.choice([1.0, 1.0, 0.95])
    if kind == "csr":
        maps = rng.choice(["sign", "gauss"])
        m = log(2000, 1_000_000 if maps == "sign" else 150_000)
        n = log(500, 100_000 if maps == "sign" else 30_000)
        return _csr(m, n, rng.randint(4, 24), rng.choice(["even", "skewed"]), maps, log(5, 70), max(m // rng.randint(1, 40), 100), nu)
    if kind == "dense":
        maps, precision = rng.choice([("gauss", "fp32"), ("gauss", "fp32"), ("gauss", "bf16"), ("gauss", "bf16"), ("sign", "fp32")])
        m, n = log(2000, 60_000), log(500, 20_000)
        return _dense(m, n, rng.choice(["col", "row"]), maps, precision, log(5, 50), min(m, log(400, 10_000)), nu)
    if kind == "rbf":
        precision = rng.choice(["fp32", "bf16"])
        m = log(2000, 30_000 if precision == "fp32" else 60_000)
        return _rbf(m, rng.randint(3, 128), precision, log(5, 64), min(m, log(500, 5000)))
    if kind == "pair":
        precision = rng.choice(["fp32", "bf16"])
        m = log(1000, 20_000 if precision == "fp32" else 50_000)
        return _pair(m, rng.randint(3, 64), rng.randint(20, 190), precision)
    if rng.random() < 0.5:
        return _approx(log(10_000, 600_000), log(2000, 60_000), "csr", log(5, 30), 10_000)
    return _approx(log(5000, 50_000), log(1000, 10_000), "dense", log(5, 50), 8192)


# ------------------------------------------------------------------- maps --
# The library's documented map generator (Philox4x32-10, Salmon et al. 2011)
# in integer torch arithmetic, for inputs and exact results made without it.
def _philox(ctr, seed):
    mask = 0xFFFFFFFF
    c, k0, k1 = list(ctr), seed & mask, 0x534B454D
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & mask) ^ c[1] ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c[3] ^ k1, p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c


def _gauss_map(seed, nrow, ncol, precision="fp32"):
    """Stored nrow x ncol values as the context holds them (FP32, or on the BF16 grid), as FP64."""
    total = nrow * ncol
    flat = torch.empty(total, dtype=torch.float64, device=DEV)
    maxval = math.sqrt(2.0 * math.log(float(total)))
    step = 1 << 25
    for e0 in range(0, total, step):
        e1 = min(total, e0 + step)
        blk = torch.arange(e0 // 2, (e1 + 1) // 2, device=DEV, dtype=torch.int64)
        tag = torch.full_like(blk, 0x47415553)
        v = _philox([blk & 0xFFFFFFFF, blk >> 32, tag, torch.zeros_like(blk)], seed)
        b = torch.stack([(v[0] << 21) | (v[1] >> 11), (v[2] << 21) | (v[3] >> 11)], 1).reshape(-1)
        u = (2 * b - (1 << 53)).double() * 2.0**-53
        x = (maxval * u).float()
        flat[e0:e1] = (x.bfloat16() if precision == "bf16" else x).double()[: e1 - e0]
    return flat.reshape(ncol, nrow).t()


def _sign_map(seed, nrow, ncol):
    """(columns, signs), zeta per stored row."""
    zeta = max(2, min(ncol, 8))
    row = torch.arange(nrow, device=DEV, dtype=torch.int64)
    tag, one = torch.full_like(row, 0x53534731), torch.ones_like(row)
    a, b, s = (_philox([row & 0xFFFFFFFF, row >> 32, tag, one * t], seed) for t in range(3))
    idx = ((torch.stack(a + b, 1)[:, :zeta] * ncol) >> 32).sort(1).values
    sgn = 1.0 - 2.0 * ((s[0][:, None] >> torch.arange(zeta, device=DEV)) & 1).double()
    return idx, sgn


def _sign_dense(seed, nrow, ncol):
    idx, sgn = _sign_map(seed, nrow, ncol)
    return torch.zeros(nrow, ncol, dtype=torch.float64, device=DEV).scatter_add_(1, idx, sgn)


def _sizes(case):
    k = 4 * case["rank"] + 1
    return k, 2 * k + 1


def _row_weights(case):
    """The weight of each row's window in X and Z: nu^(windows after it)."""
    m, w = case["m"], case["window"]
    win = torch.arange(m, device=DEV) // w
    return float(case.get("nu", 1.0)) ** ((m + w - 1) // w - 1 - win).double()


# ----------------------------------------------------------------- inputs --
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _make_csr(m, n, nnz_row, rows, seed):
    """Seeded CSR block: sorted distinct columns, N(0, 1) values on a planted low-rank part. "skewed" rows have
    log-normal lengths (some empty, some many times the mean)."""
    g = _gen(seed)
    if rows == "even":
        cnt = torch.full((m,), nnz_row, device=DEV, dtype=torch.int64)
    else:
        cnt = (nnz_row / 1.65 * torch.randn(m, generator=g, device=DEV).exp()).long().clamp_(0, min(20 * nnz_row, n // 2))
    row = torch.repeat_interleave(torch.arange(m, device=DEV), cnt)
    key = torch.unique(row * n + torch.randint(0, n, (row.numel(),), generator=g, device=DEV))
    row, col = key // n, (key % n).int()
    rowptr = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    rowptr[1:] = torch.bincount(row, minlength=m).cumsum(0)
    val = torch.randn(row.numel(), generator=g, device=DEV)
    p = 4
    u, v = torch.randn(m, p, generator=g, device=DEV), torch.randn(n, p, generator=g, device=DEV)
    for q in range(p):
        val += 2.5 * u[row, q] * v[col.long(), q]
    return rowptr, col, val


def _make_dense(m, n, layout, seed):
    """U diag(i^-1.5) V^T + 1e-4 N(0, 1), in 64 directions, FP32."""
    g = _gen(seed)
    p = min(64, m, n)
    u = torch.linalg.qr(torch.randn(m, p, generator=g, device=DEV))[0]
    v = torch.linalg.qr(torch.randn(n, p, generator=g, device=DEV))[0]
    v *= torch.arange(1, p + 1, device=DEV) ** -1.5
    if layout == "row":
        a = torch.randn(m, n, generator=g, device=DEV).mul_(1e-4)
        return a.addmm_(u, v.t())
    a = torch.randn(n, m, generator=g, device=DEV).mul_(1e-4)
    return a.addmm_(v, u.t()).t()


def _make_points(m, d, seed):
    """8-component Gaussian mixture and gamma = 1 / (2 median squared distance)."""
    g = _gen(seed)
    means = 2.0 * torch.randn(8, d, generator=g, device=DEV)
    pts = means[torch.randint(0, 8, (m,), generator=g, device=DEV)] + torch.randn(m, d, generator=g, device=DEV)
    sub = pts[:1000].double()
    return pts, 1.0 / (2.0 * float(torch.cdist(sub, sub).pow(2).median()))


def _make_pair(case, seed):
    """Points, gamma, Omega and the cotangent 2 K Omega^T (a squared-norm loss)."""
    m, k = case["m"], case["k"]
    pts, gamma = _make_points(m, case["d"], seed)
    om = torch.randn(k, m, generator=_gen(seed + 1), device=DEV)
    sq, bar = pts.square().sum(1), torch.empty(m, k, device=DEV)
    for r in range(0, m, 8192):
        d2 = (sq[r:r + 8192, None] + sq - 2.0 * (pts[r:r + 8192] @ pts.t())).clamp_min_(0)
        bar[r:r + 8192] = 2.0 * (d2.mul_(-gamma).exp_() @ om.t())
    return pts, gamma, om, bar


def _make_matrix(case, seed):
    if case["source"] == "csr":
        return _make_csr(case["m"], case["n"], 10, "even", seed)
    return _make_dense(case["m"], case["n"], "col", seed)


def _params(case):
    p = sk.AlgParams()
    p.matrix_m = case["m"]
    p.matrix_n = case.get("n", case["m"])
    p.rank, p.window, p.sketch_nu = case["rank"], case["window"], case.get("nu", 1.0)
    p.precision = {"fp32": L.PREC_FP32, "bf16": L.PREC_BF16}[case.get("precision", "fp32")]
    p.issparse = case["kind"] == "csr" or case.get("source") == "csr"
    maps = case.get("maps", "sign" if case.get("source") == "csr" else "gauss")
    p.dim_redux = L.MAP_SPARSE_SIGN if maps == "sign" else L.MAP_GAUSS
    if case["kind"] == "rbf":
        p.kernel_func, p.force_three_sketch = L.KERNEL_GAUSSRBF, True
    return p


def prepare(case, seed):
    """The input in device memory, the context with its maps and the buffers that results go to."""
    st = {"case": case}
    if case["kind"] == "pair":
        st["pts"], st["gamma"], st["om"], st["bar"] = _make_pair(case, seed)
        st["ctx"] = sk.SketchySVD(sk.AlgParams(
            matrix_m=1, matrix_n=1, precision=L.PREC_BF16 if case["precision"] == "bf16" else L.PREC_FP32))
        return st
    p = _params(case)
    if case["kind"] == "csr":
        st["A"] = _make_csr(case["m"], case["n"], case["nnz_row"], case["rows"], seed)
    elif case["kind"] == "dense":
        st["A"] = _make_dense(case["m"], case["n"], case["layout"], seed)
    elif case["kind"] == "rbf":
        st["A"], p.kernel_gamma = _make_points(case["m"], case["d"], seed)
    else:
        st["A"] = _make_matrix(case, seed)
    ctx = st["ctx"] = sk.SketchySVD(p)
    m, n, r, (k, s) = case["m"], p.matrix_n, case["rank"], _sizes(case)
    if case["kind"] == "approx":
        for which, t in zip((L.SKETCH_X, L.SKETCH_Y, L.SKETCH_Z), _sketches(case, st["A"])[0]):
            ctx.set_sketch(which, t.float().contiguous())
        st["out"] = tuple(torch.empty(q, dtype=torch.float64, device=DEV) for q in ((r, m), (r,), (r, n)))
    else:
        st["out"] = [torch.empty(q, device=DEV) for q in ((k, n), (m, k), (s, s))]
    return st


# ------------------------------------------------------------------- pass --
def run(st):
    case, ctx = st["case"], st["ctx"]
    if case["kind"] == "pair":
        y = sk.rbf_sketch_fwd(st["pts"], st["gamma"], st["om"], ctx=ctx)
        dx, dg = sk.rbf_sketch_vjp(st["pts"], st["gamma"], st["om"], st["bar"], ctx=ctx)
        return {"Y": y, "dX": dx, "dgamma": dg}
    if case["kind"] == "approx":
        u, s, v = ctx.low_rank_approx(device_out=st["out"])
        return {"U": u, "S": s, "V": v, "rnorms": ctx.residuals(st["A"], None, None, None)}
    ctx.reset()
    ctx.update_rows(st["A"])
    x, y, z = (ctx.get_sketch(w, out=t) for w, t in zip((L.SKETCH_X, L.SKETCH_Y, L.SKETCH_Z), st["out"]))
    return {"X": x, "Y": y, "Z": z}


# ------------------------------------------------------------------- work --
def work(case):
    m = case["m"]
    if case["kind"] == "pair":
        d, k = case["d"], case["k"]
        # K once per direction, K Omega^T; M = Ybar Omega, E X and E^T X
        return {"bytes": 4.0 * (2 * m * d + 3 * m * k), "flops": 2.0 * m * m * (d + k) + 2.0 * m * m * (3 * d + k)}
    k, s = _sizes(case)
    n = case.get("n", m)
    out = 4.0 * (k * n + m * k + s * s)
    if case["kind"] == "rbf":
        d = case["d"]
        return {"bytes": 4.0 * (m * d + 2 * m * (k + s)) + out, "flops": 2.0 * m * m * (d + 2 * k + s) + 2.0 * m * s * s}
    if case["kind"] == "csr":
        nnz = m * case["nnz_row"]
        if case["maps"] == "sign":
            return {"bytes": 8.0 * (m + nnz) + 32.0 * n + out, "flops": 16.0 * nnz}
        return {"bytes": 8.0 * (m + nnz) + 4.0 * (m + n) * (k + s) + out,
                "flops": 2.0 * nnz * (2 * k + s) + 2.0 * min(m, n) * s * s}
    if case["kind"] == "dense":
        if case["maps"] == "sign":  # the columns and rows that the maps name
            return {"bytes": 32.0 * (m * k + n * k + s * s) + out, "flops": 16.0 * (m * k + n * k + s * s)}
        return {"bytes": 4.0 * (m * n + (m + n) * (k + s)) + out, "flops": 2.0 * m * n * (2 * k + s) + 2.0 * m * s * s}
    r = case["rank"]
    a_bytes, a_items = (88.0 * m, 10.0 * m) if case["source"] == "csr" else (4.0 * m * n, float(m) * n)
    # a QR of Y and X^T each (R and Q), the small products, U and V; the residual pass reads A once
    return {"bytes": 4.0 * (m + n) * k + 4.0 * s * s + 8.0 * (m + n) * r + a_bytes,
            "flops": 4.0 * (m + n) * k * k + 2.0 * (m + n) * k * r + 4.0 * a_items * r}


# ------------------------------------------------------------------ exact --
def _dense64(a, m, chunk):
    for r in range(0, m, chunk):
        yield r, min(m, r + chunk), a[r:r + chunk].double()


def _kernel64(pts, gamma, r0, r1):
    p = pts.double()
    sq = p.square().sum(1)
    d2 = (sq[r0:r1, None] + sq - 2.0 * (p[r0:r1] @ p.t())).clamp_min_(0)
    i = torch.arange(r0, r1, device=DEV)
    d2[i - r0, i] = 0.0
    return d2


def _pick_rows(rowptr, rows):
    """(entry of `rows`, position in col / val) of every nonzero of the given rows."""
    cnt = rowptr[rows + 1] - rowptr[rows]
    e = torch.repeat_interleave(torch.arange(rows.numel(), device=DEV), cnt)
    first = torch.cumsum(cnt, 0) - cnt
    return e, rowptr[rows][e] + torch.arange(e.numel(), device=DEV) - first[e]


def _sketches(case, a, gamma=None):
    """(X, Y, Z) in FP64 and the maps Phi~ (s x m) and Psi~ (s x n) as (values, transposed dense) makers."""
    m, n, (k, s) = case["m"], case.get("n", case["m"]), _sizes(case)
    wt = _row_weights(case)
    csr = case["kind"] == "csr" or case.get("source") == "csr"
    sign = case.get("maps", "sign" if case.get("source") == "csr" else "gauss") == "sign"
    prec = case.get("precision", "fp32")
    z64 = dict(dtype=torch.float64, device=DEV)
    if csr:
        rowptr, col, val = a
        row = torch.repeat_interleave(torch.arange(m, device=DEV), rowptr[1:] - rowptr[:-1])
        j, v = col.long(), val.double()
    if csr and sign:
        oi, os = _sign_map(1, n, k)
        pi, ps = _sign_map(3, n, s)
        y = torch.zeros(m * k, **z64)
        for t in range(oi.shape[1]):
            y.index_add_(0, row * k + oi[j, t], v * os[j, t])
        x, z = torch.zeros(k * n, **z64), torch.zeros(s * s, **z64)
        ui, us = _sign_map(0, k, m)
        e, p = _pick_rows(rowptr, ui.reshape(-1))
        w = us.reshape(-1)[e] * wt[ui.reshape(-1)[e]] * v[p]
        x.index_add_(0, e // ui.shape[1] * n + j[p], w)
        fi, fs = _sign_map(2, s, m)
        e, p = _pick_rows(rowptr, fi.reshape(-1))
        w = fs.reshape(-1)[e] * wt[fi.reshape(-1)[e]] * v[p]
        for t in range(pi.shape[1]):
            z.index_add_(0, e // fi.shape[1] * s + pi[j[p], t], w * ps[j[p], t])
        return (x.reshape(k, n), y.reshape(m, k), z.reshape(s, s)), (fi, fs), (pi, ps)
    if csr:  # all four maps stored with the long dimension first
        a64 = torch.sparse_csr_tensor(rowptr, j, v, size=(m, n))
        aw = torch.sparse_coo_tensor(torch.stack([j, row]), v * wt[row], size=(n, m)).coalesce()
        y = a64 @ _gauss_map(1, n, k).contiguous()
        x = torch.sparse.mm(aw, _gauss_map(0, m, k).contiguous()).t()
        t = a64 @ _gauss_map(3, n, s).contiguous()
        return (x, y, _gauss_map(2, m, s).t() @ (t * wt[:, None])), None, None
    make = _sign_dense if sign else lambda q, nr, nc: _gauss_map(q, nr, nc, prec)
    u, o, f, p = make(0, k, m), make(1, k, n), make(2, s, m), make(3, s, n)
    x, y, z = torch.zeros(k, n, **z64), torch.empty(m, k, **z64), torch.zeros(s, s, **z64)
    chunk = max(256, min(m, 200_000_000 // n))
    blocks = _dense64(a, m, chunk) if gamma is None else (
        (r, min(m, r + chunk), _kernel64(a, gamma, r, min(m, r + chunk)).mul_(-gamma).exp_()) for r in range(0, m, chunk))
    for r0, r1, b in blocks:
        y[r0:r1] = b @ o.t()
        w = wt[r0:r1]
        x += (u[:, r0:r1] * w) @ b
        z += (f[:, r0:r1] * w) @ (b @ p.t())
    return (x, y, z), f, p


def _exact_pair(case, seed):
    pts, gamma, om, bar = _make_pair(case, seed)
    m, p, o = case["m"], pts.double(), om.double()
    y = torch.empty(m, case["k"], dtype=torch.float64, device=DEV)
    rows, cols, ex, dg = torch.empty(m, **_F64), torch.zeros(m, **_F64), torch.zeros_like(p), 0.0
    chunk = max(256, 200_000_000 // m)
    for r in range(0, m, chunk):
        e = min(m, r + chunk)
        d2 = _kernel64(pts, gamma, r, e)
        kk = (d2 * -gamma).exp_()
        y[r:e] = kk @ o.t()
        kk *= bar[r:e].double() @ o
        i = torch.arange(r, e, device=DEV)
        kk[i - r, i] = 0.0
        dg -= float((kk * d2).sum())
        rows[r:e] = kk.sum(1)
        cols += kk.sum(0)
        ex[r:e] += kk @ p
        ex += kk.t() @ p[r:e]
    return {"Y": y, "dX": -2.0 * gamma * ((rows + cols)[:, None] * p - ex), "dgamma": dg}


_F64 = dict(dtype=torch.float64, device=DEV)


def _exact_approx(case, seed):
    """Singular values and residual norms; the vectors' signs are free."""
    a, r = _make_matrix(case, seed), case["rank"]
    (x, y, z), f, p = _sketches(case, a)
    x, y, z = x.float().double(), y.float().double(), z.float().double()
    pq, q = torch.linalg.qr(x.t())[0], torch.linalg.qr(y)[0]

    def apply(mp, b):
        if not isinstance(mp, tuple):
            return mp @ b
        idx, sgn = mp  # stored s x m: rows of b gathered; stored n x s: scattered
        if idx.shape[0] == z.shape[0]:
            return sum(sgn[:, t, None] * b[idx[:, t]] for t in range(idx.shape[1]))
        out = torch.zeros(z.shape[0], b.shape[1], **_F64)
        for t in range(idx.shape[1]):
            out.index_add_(0, idx[:, t], sgn[:, t, None] * b)
        return out

    u1, t1 = torch.linalg.qr(apply(f, q))
    u2, t2 = torch.linalg.qr(apply(p, pq))
    core = torch.linalg.solve_triangular(t1, u1.t() @ z @ u2, upper=True)
    core = torch.linalg.solve_triangular(t2, core.t(), upper=True).t()
    uc, s, vt = torch.linalg.svd(core)
    u, s, v = (q @ uc)[:, :r], s[:r], (pq @ vt.t())[:, :r]
    if isinstance(a, tuple):
        a64 = torch.sparse_csr_tensor(a[0], a[1].long(), a[2].double(), size=(case["m"], case["n"]))
        row = torch.repeat_interleave(torch.arange(case["m"], device=DEV), a[0][1:] - a[0][:-1])
        at = torch.sparse_coo_tensor(torch.stack([a[1].long(), row]), a[2].double(), size=(case["n"], case["m"])).coalesce()
        av, atu = a64 @ v.contiguous(), torch.sparse.mm(at, u.contiguous())
    else:
        av, atu = torch.empty_like(u), torch.zeros_like(v)
        for r0, r1, b in _dense64(a, case["m"], max(256, 200_000_000 // case["n"])):
            av[r0:r1] = b @ v
            atu += b.t() @ u[r0:r1]
    rn = ((av - u * s).square().sum(0) + (atu - v * s).square().sum(0)).sqrt()
    return {"U": None, "S": s, "V": None, "rnorms": rn}


def exact(case, seed):
    if case["kind"] == "pair":
        return _exact_pair(case, seed)
    if case["kind"] == "approx":
        return _exact_approx(case, seed)
    gamma = None
    if case["kind"] == "csr":
        a = _make_csr(case["m"], case["n"], case["nnz_row"], case["rows"], seed)
    elif case["kind"] == "dense":
        a = _make_dense(case["m"], case["n"], case["layout"], seed)
    else:
        a, gamma = _make_points(case["m"], case["d"], seed)
    x, y, z = _sketches(case, a, gamma)[0]
    return {"X": x, "Y": y, "Z": z}
