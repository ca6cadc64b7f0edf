"""Calls that follow one another without a synchronise, and handles whose calls
were not ordered: what the kernels leave behind for the next launch."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

COL = 0


@pytest.fixture(scope="module")
def mp():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from drb import mp as _mp
    return _mp


def powerlaw(mp, m, mean, cap, dtype, seed=3):
    import drb
    rp, ci, v = drb.gen.powerlaw_csr(m, m, alpha=drb.gen.zipf_alpha_for_mean(1, cap, mean), hi=cap,
                                     seed=seed, value_dtype=dtype)
    return mp.distributed_sparse_matrix(mp.csr_matrix_view(v, rp, ci, (m, m)), 0)


@pytest.mark.parametrize("m", [300, 40_000])
def test_unordered_calls_leave_the_handle_usable(mp, m):
    """One handle's calls must be stream-ordered.  Where a program breaks that,
    their results are undefined, but later, ordered calls are right again: the
    work counter is back at zero whatever the grids that shared it."""
    a = powerlaw(mp, m, 12, 4096 if m > 4096 else 64, np.float32)
    assert a.variant() != 2048  # the kernels with a work counter
    x = torch.rand(m, device="cuda")
    b = torch.rand(m, device="cuda")
    want = torch.zeros(m, device="cuda")
    a.gemv_device(x, want, 1, COL)
    torch.cuda.synchronize()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    y1, y2, y = (torch.zeros(m, device="cuda") for _ in range(3))
    for rep in range(20):
        for _ in range(5):
            a.gemv_device(x, y1, 1, COL, stream=s1)
            mp.residual_norm2(a, x, b, y2, stream=s2)  # another grid on the same counter
        torch.cuda.synchronize()
        y.zero_()
        a.gemv_device(x, y, 1, COL)
        assert torch.equal(y, want), rep


def chain(steps, one, paused):
    """`steps` calls of one(i), each reading what the last wrote; paused: the GPU
    is idle before every call."""
    for i in range(steps):
        if paused:
            torch.cuda.synchronize()
        one(i)
    torch.cuda.synchronize()


def same_chained_and_paused(make):
    """The calls of a chain overlap their launches; their results are those of
    calls that start on an idle GPU, bit for bit."""
    results = []
    for paused in (True, False, False):
        outs, steps, one = make()
        chain(steps, one, paused)
        results.append([o.clone() for o in outs])
    for other in results[1:]:
        for u, v in zip(results[0], other):
            assert torch.isfinite(u).all()
            assert torch.equal(u, v)


@pytest.mark.parametrize("kind,dtype,env", [
    ("band", np.float32, {}), ("band", np.float64, {}),
    ("powerlaw", np.float32, {"DRB_SPMV_VARIANT": "128,1"}),
    ("powerlaw", np.float32, {"DRB_SPMV_VARIANT": "256,1,1"}),
    ("powerlaw", np.float64, {}), ("powerlaw", np.float64, {"DRB_COLSPLIT": "3"})])
def test_products_feed_the_next_product(mp, kind, dtype, env, monkeypatch):
    import drb
    for key, value in env.items():
        monkeypatch.setenv(key, value)
    m = 30_000
    if kind == "band":
        rp = np.arange(0, 5 * m + 1, 5).astype(np.int32)
        ci = ((np.arange(m)[:, None] + np.array([-7, -1, 0, 1, 7])) % m).astype(np.int32)
        ci = np.sort(ci, 1).reshape(-1)
        v = drb.gen.values(5 * m, seed=1, dtype=dtype)
    else:
        rp, ci, v = drb.gen.powerlaw_csr(m, m, alpha=drb.gen.zipf_alpha_for_mean(1, 8192, 10),
                                         hi=8192, seed=2, value_dtype=dtype)
    rows = np.repeat(np.arange(m), np.diff(rp))
    total = np.bincount(rows, np.abs(v), minlength=m)
    v = (v * (2.0 / total[rows])).astype(dtype)  # products keep their size
    a = mp.distributed_sparse_matrix(mp.csr_matrix_view(v, rp, ci, (m, m)), 0)
    assert (a.variant() == 2048) == (kind == "band")
    x0 = torch.from_numpy(drb.gen.values(m, seed=3, dtype=dtype)).cuda()

    def make():
        x, norms = [x0.clone(), torch.zeros_like(x0)], torch.zeros(60, dtype=torch.float64,
                                                                  device="cuda")

        def one(i):
            a.gemv_device(x[i % 2], x[1 - i % 2], 1, COL)
            mp.dot(x[1 - i % 2], x[1 - i % 2], norms[i:i + 1])
        return [x[0], x[1], norms], 60, one
    same_chained_and_paused(make)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,k", [(300, 1), (301, 1), (1200, 1), (2101, 1), (2304, 1), (300, 3),
                                 (301, 20), (1200, 12), (1201, 5)])
def test_dense_products_and_reductions_feed_one_another(mp, dtype, n, k):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    A = torch.randn(n, n, generator=g, device="cuda", dtype=dtype) * (n ** -0.5)
    x0 = torch.randn(n * k, generator=g, device="cuda", dtype=dtype)

    def make():
        x = [x0.clone(), torch.zeros_like(x0)]
        dots = torch.zeros(40, dtype=torch.float64, device="cuda")
        top = torch.zeros(40, dtype=dtype, device="cuda")
        last = torch.zeros(1, dtype=dtype, device="cuda")

        def one(i):
            mp.dense_gemv(A, x[i % 2], x[1 - i % 2], k, COL)
            mp.dot(x[i % 2], x[1 - i % 2], dots[i:i + 1])
            mp.reduce(x[1 - i % 2], 0.0, max, out=top[i:i + 1])
            mp.reduce(top, 0.0, max, out=last)
        return [x[0], x[1], dots, top, last], 40, one
    same_chained_and_paused(make)


def test_current_stream_without_the_private_calls(mp, monkeypatch):
    side = torch.cuda.Stream()
    for stream in (torch.cuda.default_stream(), side):
        with torch.cuda.stream(stream):
            fast = mp._stream()
            with monkeypatch.context() as patch:
                patch.setattr(mp, "_RAW_STREAM", None)
                assert mp._stream() == fast == stream.cuda_stream
