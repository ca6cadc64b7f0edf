"""Performance cases of the gemv path: what its users call, over the sizes they call it at.

listed()            the fixed cases
draw(rng)           one more case of the same ranges
prepare(case, seed) what a program holds before the call: handles, plans, vectors on the GPU
run(state)          one pass through the public entry points of drb.mp; returns its outputs
work(case)          the bytes and operations of one pass that cannot be avoided
exact(case, seed)   the same outputs in 64-bit arithmetic, in plain torch

Matrices, vectors and right-hand sides are made on the GPU from the seed
alone, the way the benchmark's are: power-law (truncated Zipf) or bounded row
lengths with uniform columns, bands, 5-point Laplacians; values
U(-1, 1), dense operands N(0, 1).
"""
import functools
import math
import operator
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "distributed-ranges_b200"))

from drb import _capi as capi  # noqa: E402
from drb import mp  # noqa: E402

_DT = {"f32": torch.float32, "f64": torch.float64, "bf16": torch.bfloat16}
_BYTES = {"f32": 4, "f64": 8, "bf16": 2}
_LAYOUT = {"col": capi.DRB_COL_MAJOR, "row": capi.DRB_ROW_MAJOR}


def listed():
    return [
        # The reference's own use at its tests' size: a banded 1000 x 1000 FP64
        # matrix, x broadcast, the result wanted on the host.  Call overhead.
        dict(name="gemv_band_host", kind="gemv", pattern="band", m=1000, n=1000, mean=41.0, cap=41,
             dtype="f64", x="f64", host=True, compensated=False),
        # A regular mid-size matrix (131072^2, 16 per row), device resident: one
        # step of an explicit time loop.  Microseconds, all of it in L2.
        dict(name="gemv_fixed16_f32", kind="gemv", pattern="fixed", m=131072, n=131072, mean=16.0,
             cap=16, dtype="f32", x="f32", host=False, compensated=False),
        # A large graph matrix whose x (54 MB) does not stay in L2, with rows up
        # to 16384 nonzeros: one PageRank-like step.
        dict(name="gemv_powerlaw_f32", kind="gemv", pattern="powerlaw", m=13421773, n=13421773,
             mean=8.0, cap=16384, dtype="f32", x="f32", host=False, compensated=False),
        # BF16 storage with f32 x and compensated sums, rows up to 65536.
        dict(name="gemv_powerlaw_bf16", kind="gemv", pattern="powerlaw", m=2097152, n=2097152,
             mean=32.0, cap=65536, dtype="bf16", x="f32", host=False, compensated=False),
        # A slim matrix of 20 columns (the reference tests' width), column-major:
        # a block of vectors through one sparse operator.
        dict(name="slim20_f32", kind="slim", m=1000003, n=1000003, lo=8, hi=64, k=20, dtype="f32",
             x="f32", layout="col"),
        # Fused residual and adjoint of a sparse least-squares step: forward and
        # backward, gradients for x and for every stored value.
        dict(name="residual_backward_f64", kind="adjoint", pattern="powerlaw", m=1500007, n=1500007,
             mean=20.0, cap=16384, dtype="f64"),
        # An inner solver with a fixed budget of iterations on a 5-point Laplacian.
        dict(name="cg_laplacian_f64", kind="cg", g=1024, iters=64, dtype="f64"),
        # Dense gemv of a square matrix, one right-hand side.
        dict(name="dense_f32", kind="dense", m=8192, n=8192, k=1, dtype="f32", layout="col", pad=0),
        # Dense gemv with odd sizes and several right-hand sides.
        dict(name="dense_ragged_f64", kind="dense", m=5003, n=3001, k=20, dtype="f64", layout="col",
             pad=0),
        # Dense BF16 products with 32 right-hand sides, ragged square sizes, one
        # plan over all matrices.
        dict(name="dense_batch_bf16", kind="dense_batch", count=16, lo=256, hi=8192, k=32,
             layout="col"),
        # Many sparse matrices with 16 right-hand sides each in one launch.
        dict(name="batch_spmm_f32", kind="batch", count=16, rows=102400, lo=8, hi=64, k=16,
             dtype="f32", x="f32", layout="col"),
        # The vector side of an iterative method: a dot product, a sum and a
        # maximum over a long vector.
        dict(name="vectors_f32", kind="vector", n=10000019, dtype="f32"),
    ]


# ---- drawn cases -----------------------------------------------------------------


def _log(rng, lo, hi):
    """An integer of [lo, hi], uniform in its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_gemv(rng):
    pattern = rng.choice(["powerlaw", "powerlaw", "uniform", "fixed", "band"])
    dtype = rng.choice(["f32", "f32", "f64", "bf16"])
    mean = float(_log(rng, 3, 48))
    m = _log(rng, 1000, int(min(13e6, 100e6 / mean)))
    n = m if rng.random() < 0.6 else _log(rng, max(1000, m // 8), min(13_000_000, 8 * m))
    cap = {"powerlaw": min(_log(rng, 1024, 65536), n // 4), "uniform": int(2 * mean),
           "fixed": int(mean), "band": int(mean)}[pattern]
    if pattern == "band":
        n = m
    return dict(kind="gemv", pattern=pattern, m=m, n=n, mean=mean, cap=max(cap, int(4 * mean)
                if pattern == "powerlaw" else cap), dtype=dtype,
                x="f32" if dtype == "bf16" and rng.random() < 0.7 else dtype,
                host=m < 2_000_000 and rng.random() < 0.2,
                compensated=dtype == "f32" and rng.random() < 0.2)


def _draw_slim(rng):
    dtype = rng.choice(["f32", "f32", "f64", "bf16"])
    k = _log(rng, 2, 40)
    lo = rng.randint(1, 16)
    hi = lo + _log(rng, 4, 64)
    top = 700e6 / (k * (lo + hi) / 2) / (_BYTES[dtype] / 4 if dtype == "f64" else 1)
    m = _log(rng, 1000, int(min(2e6, top)))
    return dict(kind="slim", m=m, n=m if rng.random() < 0.6 else _log(rng, max(1000, m // 4), 4 * m),
                lo=lo, hi=hi, k=k, dtype=dtype,
                x="f32" if dtype == "bf16" and rng.random() < 0.5 else dtype,
                layout=rng.choice(["col", "col", "row"]))


def _draw_adjoint(rng):
    dtype = rng.choice(["f32", "f64"])
    if rng.random() < 0.35:
        g = _log(rng, 550, 1600)
        return dict(kind="adjoint", pattern="laplacian", m=g * g, n=g * g, mean=5.0, cap=5, dtype=dtype)
    mean = float(_log(rng, 5, 40))
    m = _log(rng, 300000, int(min(2.5e6, 30e6 / mean)))
    return dict(kind="adjoint", pattern=rng.choice(["powerlaw", "uniform"]), m=m,
                n=_log(rng, m // 2, 2 * m), mean=mean, cap=_log(rng, 1024, 16384), dtype=dtype)


def _draw_cg(rng):
    return dict(kind="cg", g=_log(rng, 48, 1500), iters=rng.randint(20, 64),
                dtype=rng.choice(["f32", "f64"]))


def _draw_dense(rng):
    m = _log(rng, 64, 16384)
    n = _log(rng, 64, min(16384, (1 << 26) // m))
    if rng.random() < 0.5:
        n = max(64, n // 32 * 32)
    k = 1 if rng.random() < 0.4 else _log(rng, 2, 32)
    return dict(kind="dense", m=m, n=n, k=k, dtype=rng.choice(["f32", "f64"]),
                layout=rng.choice(["col", "row"]), pad=rng.choice([0, 0, 8]))


def _draw_dense_batch(rng):
    count = _log(rng, 1, 32)
    hi = _log(rng, 256, min(8192, int(math.sqrt(1.2e9 / count))))
    return dict(kind="dense_batch", count=count, lo=max(64, hi // rng.choice([1, 2, 32])), hi=hi,
                k=_log(rng, 1, 128), layout=rng.choice(["col", "row"]))


def _draw_batch(rng):
    dtype = rng.choice(["f32", "f32", "f64", "bf16"])
    count = _log(rng, 2, 64)
    k = _log(rng, 1, 32)
    lo = rng.randint(1, 12)
    hi = lo + _log(rng, 4, 64)
    top = 900e6 / (count * k * (lo + hi) / 2) / (2 if dtype == "f64" else 1)
    return dict(kind="batch", count=count, rows=_log(rng, 500, int(max(1000, min(200000, top)))),
                lo=lo, hi=hi, k=k, dtype=dtype,
                x="f32" if dtype == "bf16" and rng.random() < 0.5 else dtype,
                layout=rng.choice(["col", "col", "row"]))


def _draw_vector(rng):
    return dict(kind="vector", n=_log(rng, 1000, 100_000_000), dtype=rng.choice(["f32", "f64"]))


def draw(rng):
    return rng.choice([_draw_gemv, _draw_gemv, _draw_slim, _draw_adjoint, _draw_cg, _draw_dense,
                       _draw_dense_batch, _draw_batch, _draw_vector])(rng)


# ---- inputs from the seed ----------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(n, dtype, g):
    return torch.rand(n, generator=g, device="cuda", dtype=dtype) * 2 - 1


@functools.lru_cache(maxsize=64)
def _zipf_cdf(mean, cap):
    """Distribution function of the Zipf law on [1, cap] whose mean is `mean`."""
    k = np.arange(1, cap + 1, dtype=np.float64)
    lo, hi = -4.0, 8.0
    for _ in range(60):
        a = 0.5 * (lo + hi)
        w = np.exp(-a * np.log(k))
        lo, hi = (a, hi) if (w * k).sum() / w.sum() > mean else (lo, a)
    w = np.exp(-0.5 * (lo + hi) * np.log(k))
    return np.cumsum(w) / w.sum()


def _row_lengths(pattern, m, mean, cap, g):
    """Row lengths: the law's m evenly spaced quantiles in a random order (so a
    case has the same number of nonzeros whatever the seed)."""
    if pattern == "fixed":
        return torch.full((m,), int(mean), device="cuda")
    if pattern == "powerlaw":
        cdf = torch.from_numpy(_zipf_cdf(mean, cap)).cuda()
        u = (torch.arange(m, device="cuda", dtype=torch.float64) + 0.5) / m
        lengths = (torch.searchsorted(cdf, u) + 1).clamp_(max=cap)
    else:
        lengths = 1 + torch.arange(m, device="cuda") % max(1, int(2 * mean) - 1)
    return lengths[torch.randperm(m, generator=g, device="cuda")]


def _scattered(lengths, n, g):
    """(rowptr, colind): uniform columns, sorted within a row (the few repeats,
    which CSR allows, stay)."""
    m = lengths.numel()
    rows = torch.repeat_interleave(torch.arange(m, device="cuda"), lengths)
    key = rows * n + torch.randint(0, n, (rows.numel(),), generator=g, device="cuda")
    key = torch.sort(key).values
    rowptr = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = lengths.cumsum(0)
    return rowptr, (key - rows * n).to(torch.int32)


def _band(m, n, width):
    """`width` neighbouring columns around the diagonal, clipped to the matrix."""
    r = torch.arange(m, device="cuda").unsqueeze(1)
    c = r - width // 2 + torch.arange(width, device="cuda")
    ok = (c >= 0) & (c < n)
    rowptr = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = ok.sum(1).cumsum(0)
    return rowptr, c[ok].to(torch.int32)


def _laplacian(gr, dtype):
    """5-point Laplacian of a gr x gr grid with zero boundary values."""
    m = gr * gr
    r = torch.arange(m, device="cuda")
    i, j = r // gr, r % gr
    cols = torch.stack([r - gr, r - 1, r, r + 1, r + gr], 1)
    ok = torch.stack([i > 0, j > 0, i >= 0, j < gr - 1, i < gr - 1], 1)
    v = torch.tensor([-1.0, -1.0, 4.0, -1.0, -1.0], device="cuda", dtype=dtype).expand(m, 5)
    rowptr = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = ok.sum(1).cumsum(0)
    return rowptr, cols[ok].to(torch.int32), v[ok]


def _csr(c, g):
    """The case's matrix on the GPU: rowptr (int64), colind (int32), values."""
    dt = torch.float64 if c["dtype"] == "f64" else torch.float32
    m, n = c["m"], c["n"]
    if c["kind"] in ("slim", "batch"):
        lengths = c["lo"] + torch.arange(m, device="cuda") % (c["hi"] - c["lo"] + 1)
        rp, ci = _scattered(lengths[torch.randperm(m, generator=g, device="cuda")], n, g)
    elif c["pattern"] == "band":
        rp, ci = _band(m, n, int(c["mean"]))
    elif c["pattern"] == "laplacian":
        return _laplacian(math.isqrt(m), dt)
    else:
        rp, ci = _scattered(_row_lengths(c["pattern"], m, c["mean"], c["cap"], g), n, g)
    return rp, ci, _uniform(ci.numel(), dt, g)


def _matrices(c, g):
    """The sparse matrices of a case (one, or `count` for a batch), one by one."""
    if c["kind"] != "batch":
        yield _csr(c, g), c["m"], c["n"]
        return
    for i in range(c["count"]):
        m = max(1, c["rows"] - 37 * (i % 5))  # neighbours of one size, none equal
        yield _csr(dict(c, m=m, n=m), g), m, m


def _handle(c, csr, m, n, adjoint=False):
    rp, ci, v = csr
    view = mp.csr_matrix_view(v.cpu().numpy(), rp.to(torch.int32).cpu().numpy(), ci.cpu().numpy(),
                              (m, n))
    return mp.distributed_sparse_matrix(
        view, 0, distr=mp.csr_row_distribution, adjoint=adjoint,
        storage=torch.bfloat16 if c["dtype"] == "bf16" else None, x_dtype=_DT[c.get("x", c["dtype"])],
        compensated=c.get("compensated", False))


def _x(c, count, g):
    """`count` elements of x in the type that the product reads."""
    dt = torch.float64 if c["dtype"] == "f64" else torch.float32
    return _uniform(count, dt, g).to(_DT[c.get("x", c["dtype"])])


def _ydt(c):
    return torch.float64 if c["dtype"] == "f64" else torch.float32


def _dense(c, g):
    dt = _DT[c["dtype"]]
    A = torch.randn(c["m"], c["n"] + c["pad"], generator=g, device="cuda", dtype=dt)[:, :c["n"]]
    return A, torch.randn(c["n"] * c["k"], generator=g, device="cuda", dtype=dt)


def _dense_sides(c):
    """Side lengths spread over [lo, hi], odd ones among them, in a mixed order."""
    n = c["count"]
    return [c["lo"] + (c["hi"] - c["lo"]) * ((7 * i + 3) % n + 1) // n for i in range(n)]


def _dense_mats(c, g):
    for s in _dense_sides(c):
        lda = -(-s // 8) * 8
        A = torch.randn(s, lda, generator=g, device="cuda").bfloat16()[:, :s]
        yield A, torch.randn(s * c["k"], generator=g, device="cuda").bfloat16()


# ---- prepare and run -----------------------------------------------------------------


def prepare(case, seed):
    c, g = dict(case), _gen(seed)
    s = {"kind": c["kind"], "case": c}
    kind = c["kind"]
    if kind == "gemv":
        s["a"] = _handle(c, _csr(c, g), c["m"], c["n"])
        s["b"] = mp.broadcasted_vector()
        s["b"].broadcast_data(c["n"], 0, _x(c, c["n"], g))
        s["y"] = (np.zeros(c["m"], np.float64 if c["dtype"] == "f64" else np.float32) if c["host"]
                  else torch.zeros(c["m"], dtype=_ydt(c), device="cuda"))
    elif kind == "slim":
        s["a"] = _handle(c, _csr(c, g), c["m"], c["n"])
        x = _x(c, c["n"] * c["k"], g)
        s["y"] = torch.zeros(c["m"] * c["k"], dtype=_ydt(c), device="cuda")
        s["x"] = x
    elif kind == "adjoint":
        s["a"] = _handle(c, _csr(c, g), c["m"], c["n"], adjoint=True)
        dt = _ydt(c)
        s["x"], s["b"] = _x(c, c["n"], g), _x(c, c["m"], g)
        s["y"] = torch.zeros(c["m"], dtype=dt, device="cuda")
        s["xbar"] = torch.zeros(c["n"], dtype=dt, device="cuda")
        s["abar"] = torch.zeros(s["a"].nnz(), dtype=dt, device="cuda")
    elif kind == "cg":
        m = c["g"] ** 2
        s["a"] = _handle(c, _laplacian(c["g"], _DT[c["dtype"]]), m, m)
        s["b"] = _uniform(m, _DT[c["dtype"]], g)
        s["x"] = torch.zeros(m, dtype=_DT[c["dtype"]], device="cuda")
    elif kind == "dense":
        s["A"], s["x"] = _dense(c, g)
        s["y"] = torch.zeros(c["m"] * c["k"], dtype=_DT[c["dtype"]], device="cuda")
    elif kind == "dense_batch":
        As, xs = zip(*_dense_mats(c, g))
        s["ys"] = [torch.zeros(a.shape[0] * c["k"], device="cuda") for a in As]
        s["plan"] = mp.dense_batch(As, xs, s["ys"], c["k"], _LAYOUT[c["layout"]])
    elif kind == "batch":
        s["mats"], sizes = [], []
        for csr, m, n in _matrices(c, g):
            s["mats"].append(_handle(c, csr, m, n))
            sizes.append((m, n))
        s["xs"] = [_x(c, n * c["k"], g) for _, n in sizes]
        s["ys"] = [torch.zeros(m * c["k"], dtype=_ydt(c), device="cuda") for m, _ in sizes]
        s["plan"] = mp.batch(s["mats"], c["k"], _LAYOUT[c["layout"]])
        s["plan"].bind(s["xs"], s["ys"])
    else:
        dt = _DT[c["dtype"]]
        s["u"], s["v"] = _uniform(c["n"], dt, g), _uniform(c["n"], dt, g)
        s["dot"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        s["sum"], s["max"] = (torch.zeros(1, dtype=dt, device="cuda") for _ in range(2))
    return s


def run(s):
    kind, c = s["kind"], s["case"]
    if kind == "gemv":
        mp.gemv(0, s["y"], s["a"], s["b"])
        return s["y"]
    if kind == "slim":
        s["a"].gemv_device(s["x"], s["y"], c["k"], _LAYOUT[c["layout"]])
        return s["y"]
    if kind == "adjoint":
        norm2 = mp.residual_norm2(s["a"], s["x"], s["b"], s["y"])
        s["y"].sub_(s["b"])  # the gradient of half the squared residual
        mp.gemv_backward(s["a"], s["y"], s["x"], s["xbar"], s["abar"])
        return {"norm2": norm2, "xbar": s["xbar"], "abar": s["abar"]}
    if kind == "cg":
        s["x"].zero_()
        info = mp.conjugate_gradient(s["a"], s["b"], s["x"], max_iters=c["iters"], rtol=0.0)
        return {"x": s["x"], "iterations": info["iterations"]}
    if kind == "dense":
        mp.dense_gemv(s["A"], s["x"], s["y"], c["k"], _LAYOUT[c["layout"]])
        return s["y"]
    if kind in ("dense_batch", "batch"):
        s["plan"].gemv()
        return s["ys"]
    mp.dot(s["u"], s["v"], s["dot"])
    mp.reduce(s["u"], 0.5, operator.add, out=s["sum"])
    mp.reduce(s["v"], -2.0, max, out=s["max"])
    return [s["dot"], s["sum"], s["max"]]


# ---- what a pass cannot do without -----------------------------------------------------


def _nnz(c):
    if c["kind"] in ("slim", "batch"):
        rows = c["m"] if c["kind"] == "slim" else c["count"] * c["rows"]
        return rows * (c["lo"] + c["hi"]) / 2
    return c["m"] * c["mean"]


def work(case):
    c = dict(case)
    kind, k = c["kind"], c.get("k", 1)
    vb = _BYTES[c.get("dtype", "bf16")]
    xb, yb = _BYTES[c.get("x", c.get("dtype", "bf16"))], 8 if c.get("dtype") == "f64" else 4
    if kind in ("gemv", "slim"):
        z = _nnz(c)
        return {"bytes": z * (vb + 4) + 4 * (c["m"] + 1) + k * (xb * c["n"] + yb * c["m"]),
                "flops": 2 * z * k}
    if kind == "adjoint":
        # forward: matrix, x, b -> y; backward: A^T's matrix, ybar -> xbar; columns, ybar, x -> abar
        z, m, n = _nnz(c), c["m"], c["n"]
        return {"bytes": 2 * (z * (vb + 4) + 4 * m) + z * (vb + 4) + vb * (5 * m + 3 * n) + vb * m,
                "flops": 5 * z}
    if kind == "cg":
        # matrix and p -> q, then x, r, p, q -> x, r and r, p -> p, per iteration
        m = c["g"] ** 2
        return {"bytes": c["iters"] * (5 * m * (vb + 4) + 4 * m + vb * m * 11),
                "flops": c["iters"] * m * 20}
    if kind == "dense":
        return {"bytes": vb * (c["m"] * c["n"] + k * (c["m"] + c["n"])),
                "flops": 2 * c["m"] * c["n"] * k}
    if kind == "dense_batch":
        sides = _dense_sides(c)
        return {"bytes": sum(2 * s * s + 6 * s * k for s in sides),
                "flops": sum(2 * s * s * k for s in sides)}
    if kind == "batch":
        z, rows = _nnz(c), c["count"] * c["rows"]
        return {"bytes": z * (vb + 4) + 4 * rows + k * rows * (xb + yb), "flops": 2 * z * k}
    return {"bytes": vb * 4 * c["n"], "flops": 4 * c["n"]}


# ---- the same outputs in 64 bits ---------------------------------------------------------


def _stored(v, c):
    """The values as the storage type holds them, in 64 bits."""
    return (v.bfloat16() if c["dtype"] == "bf16" else v).double()


def _product(csr, m, n, x):
    rp, ci, v = csr
    return torch.sparse_csr_tensor(rp, ci.long(), v, size=(m, n)) @ x


def _columns(x, n, k, layout):
    return x.double().reshape(k, n).t() if layout == "col" else x.double().reshape(n, k)


def _flat(y, layout):
    return (y.t() if layout == "col" else y).contiguous().reshape(-1)


def _exact_sparse(c, csr, m, n, x):
    rp, ci, v = csr
    csr = (rp, ci, _stored(v, c))
    k, layout = c.get("k", 1), c.get("layout", "col")
    return _flat(_product(csr, m, n, _columns(x, n, k, layout)), layout)


def exact(case, seed):
    c, g = dict(case), _gen(seed)
    kind = c["kind"]
    if kind in ("gemv", "slim"):
        csr = _csr(c, g)
        return _exact_sparse(c, csr, c["m"], c["n"], _x(c, c["n"] * c.get("k", 1), g))
    if kind == "adjoint":
        rp, ci, v = _csr(c, g)
        x, b = _x(c, c["n"], g).double(), _x(c, c["m"], g).double()
        r = _product((rp, ci, v.double()), c["m"], c["n"], x.unsqueeze(1)).squeeze(1) - b
        rows = torch.repeat_interleave(torch.arange(c["m"], device="cuda"), rp.diff())
        cols, g_rows = ci.long(), r[rows]
        xbar = torch.zeros(c["n"], dtype=torch.float64, device="cuda")
        xbar.index_add_(0, cols, v.double() * g_rows)
        return {"norm2": (r * r).sum().reshape(1), "xbar": xbar, "abar": g_rows * x[cols]}
    if kind == "cg":
        gr = c["g"]
        b = _uniform(gr * gr, _DT[c["dtype"]], g).double().reshape(gr, gr)

        def apply(p):
            q = 4 * p
            q[1:] -= p[:-1]
            q[:-1] -= p[1:]
            q[:, 1:] -= p[:, :-1]
            q[:, :-1] -= p[:, 1:]
            return q

        x, r, p = torch.zeros_like(b), b.clone(), b.clone()
        rr = (r * r).sum()
        for _ in range(c["iters"]):
            q = apply(p)
            alpha = rr / (p * q).sum()
            x += alpha * p
            r -= alpha * q
            new = (r * r).sum()
            p = r + (new / rr) * p
            rr = new
        return {"x": x.reshape(-1), "iterations": None}
    if kind == "dense":
        A, x = _dense(c, g)
        return _flat(A.double() @ _columns(x, c["n"], c["k"], c["layout"]), c["layout"])
    if kind == "dense_batch":
        return [_flat(A.double() @ _columns(x, A.shape[1], c["k"], c["layout"]), c["layout"])
                for A, x in _dense_mats(c, g)]
    if kind == "batch":
        mats = list(_matrices(c, g))
        xs = [_x(c, n * c["k"], g) for _, _, n in mats]
        return [_exact_sparse(c, csr, m, n, x) for (csr, m, n), x in zip(mats, xs)]
    dt = _DT[c["dtype"]]
    u, v = _uniform(c["n"], dt, g).double(), _uniform(c["n"], dt, g).double()
    return [(u * v).sum().reshape(1), (u.sum() + 0.5).reshape(1), v.max().clamp(min=-2.0).reshape(1)]
