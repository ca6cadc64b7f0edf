"""The one-launch conjugate-gradient loop (sliced-ELL matrices of at least 993
rows) against the oracle's recurrence, where its shape changes: around the
smallest size, one or several CTAs, a last slice that is not full, rows wider
than one load step, vectors partly in shared memory, more iterations than one
launch runs."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mp():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from drb import mp as _mp
    return _mp


def band(n, half):
    """Symmetric positive definite band matrix of 2 * half + 1 diagonals."""
    offs = np.arange(-half, half + 1)
    r = np.repeat(np.arange(n), offs.size)
    c = r + np.tile(offs, n)
    ok = (c >= 0) & (c < n)
    r, c = r[ok], c[ok]
    d = np.abs(r - c)
    v = np.where(d == 0, 2.0 * half + 0.5, -1.0 / np.maximum(d, 1))
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(r, minlength=n), out=rp[1:])
    return rp, c.astype(np.int32), v


def solve(mp, rp, ci, v, b, x0, iters, rtol=0.0):
    from drb import _capi as capi
    n = len(rp) - 1
    a = mp.distributed_sparse_matrix(mp.csr_matrix_view(v, rp, ci, (n, n)), 0)
    assert a.variant() == 2048
    bt, xt = torch.from_numpy(b).cuda(), torch.from_numpy(x0.copy()).cuda()
    c0 = capi.launch_count()
    info = mp.conjugate_gradient(a, bt, xt, max_iters=iters, rtol=rtol)
    launches = capi.launch_count() - c0
    x1 = xt.cpu().numpy()
    xt.copy_(torch.from_numpy(x0))
    assert mp.conjugate_gradient(a, bt, xt, max_iters=iters, rtol=rtol) == info
    assert np.array_equal(xt.cpu().numpy(), x1)  # repeatable bit for bit
    return x1, info, launches


@pytest.mark.parametrize("n,half,iters", [
    (992, 2, 9), (993, 2, 9), (1024, 2, 9), (1055, 1, 20), (1500, 3, 13), (2049, 20, 11),
    (5000, 31, 7), (40_001, 2, 30), (76_001, 4, 12), (300_007, 3, 9)])
def test_follows_oracle(mp, n, half, iters):
    rp, ci, v = band(n, half)
    rng = np.random.default_rng(n)
    b, x0 = rng.standard_normal(n), rng.standard_normal(n)
    x, info, launches = solve(mp, rp, ci, v, b, x0, iters)
    xo, it, rn, _, _ = oracle.cg(rp, ci, v, b, x0, iters, 0.0)
    assert info["iterations"] == it == iters
    assert np.linalg.norm(x - xo) <= 1e-12 * np.linalg.norm(xo)
    assert abs(info["residual_norm"] - rn) <= 1e-9 * rn
    assert (launches == 1) == (n > 992)


def laplacian_cg_long(b, g, iters):
    """`iters` updates from 0 on the 5-point Laplacian, in extended precision."""
    r = b.astype(np.longdouble).reshape(g, g)
    x, p, rr = np.zeros_like(r), r.copy(), (r * r).sum()
    for _ in range(iters):
        q = 4 * p
        q[1:] -= p[:-1]
        q[:-1] -= p[1:]
        q[:, 1:] -= p[:, :-1]
        q[:, :-1] -= p[:, 1:]
        alpha = rr / (p * q).sum()
        x += alpha * p
        r -= alpha * q
        new = (r * r).sum()
        p = r + new / rr * p
        rr = new
    return x.ravel()


@pytest.mark.parametrize("dtype,g,iters", [(np.float64, 1500, 4), (np.float32, 1500, 4)])
def test_vectors_partly_resident(mp, dtype, g, iters):
    import drb
    rp, ci, v = drb.gen.laplacian2d_csr(g, index_dtype=np.int32, value_dtype=dtype)
    n = g * g
    rng = np.random.default_rng(7)
    b, x0 = rng.standard_normal(n).astype(dtype), np.zeros(n, dtype)
    x, info, launches = solve(mp, rp, ci, v, b, x0, iters)
    assert launches == 1 and info["iterations"] == iters
    # (the oracle adds its dot products one by one in double: 1e-13 off here)
    xo = laplacian_cg_long(b, g, iters)
    # a few roundings per element and iteration
    u = 2.0 ** -24 if dtype == np.float32 else 2.0 ** -53
    assert float(np.sqrt(((x - xo) ** 2).sum())) <= 64 * iters * u * float(np.sqrt((xo ** 2).sum()))


def test_more_iterations_than_one_launch(mp):
    import drb
    g = 180
    rp, ci, v = drb.gen.laplacian2d_csr(g, index_dtype=np.int32, value_dtype=np.float32)
    n = g * g
    b = np.random.default_rng(3).standard_normal(n).astype(np.float32)
    # rtol 0: a float32 solve never gets there, so all 2500 updates run
    x, info, launches = solve(mp, rp, ci, v, b, np.zeros(n, np.float32), 2500)
    assert info["iterations"] == 2500 and not info["converged"] and launches == 3
    ax = oracle.gemv_row(rp, ci, v.astype(np.float64), x.astype(np.float64), n, n, 1,
                         oracle.ACC_LD)
    # the true residual of a float32 solution: eps * cond (about 1.3e4 here)
    assert np.linalg.norm(b - ax) <= 2.0 ** -23 * 1.4e4 * np.linalg.norm(b)


def laplacian_problem(mp, g, seed, dtype=np.float64):
    import drb
    rp, ci, v = drb.gen.laplacian2d_csr(g, index_dtype=np.int32, value_dtype=dtype)
    a = mp.distributed_sparse_matrix(mp.csr_matrix_view(v, rp, ci, (g * g, g * g)), 0)
    b = torch.from_numpy(np.random.default_rng(seed).standard_normal(g * g).astype(dtype)).cuda()
    return a, b


def test_threads_solve_at_the_same_time(mp):
    """Small solves share the GPU, large ones take turns: the bits of each are
    those of a solve alone."""
    import threading
    sizes = [48, 64, 300, 48, 120, 500]
    probs = [laplacian_problem(mp, g, i) for i, g in enumerate(sizes)]

    def one(a, b, stream=None):
        x = torch.zeros_like(b)
        if stream is not None:
            stream.wait_stream(torch.cuda.default_stream())
        info = mp.conjugate_gradient(a, b, x, max_iters=40, rtol=0.0, stream=stream)
        assert info["iterations"] == 40
        return x

    alone = [one(a, b) for a, b in probs]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        s = torch.cuda.Stream()
        for rep in range(15):
            if not torch.equal(one(*probs[i], stream=s), alone[i]):
                wrong.append((i, rep))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(probs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not any(t.is_alive() for t in threads) and not wrong


def test_a_solve_behind_queued_work_lets_others_pass(mp):
    import threading
    # (eight CTAs each: they fit beside the kernel that keeps the first waiting)
    (a1, b1), (a2, b2) = laplacian_problem(mp, 64, 1), laplacian_problem(mp, 64, 2)
    x1, x2 = torch.zeros_like(b1), torch.zeros_like(b2)
    for a, b, x in ((a1, b1, x1), (a2, b2, x2)):  # (allocations, module loading)
        mp.conjugate_gradient(a, b, x, max_iters=2, rtol=0.0)
    torch.cuda.synchronize()
    s1, s2, busy = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(s1):
        torch.cuda._sleep(3_000_000_000)  # over a second, one thread
        busy.record(s1)
    waiting = threading.Thread(
        target=lambda: mp.conjugate_gradient(a1, b1, x1, max_iters=20, rtol=0.0, stream=s1))
    waiting.start()
    import time
    time.sleep(0.1)  # it has called by now
    mp.conjugate_gradient(a2, b2, x2, max_iters=20, rtol=0.0, stream=s2)
    assert not busy.query()
    waiting.join(60)
    assert not waiting.is_alive()


@pytest.mark.parametrize("n,half", [(993, 2), (5000, 31), (300_007, 3)])
@pytest.mark.parametrize("absent", [0, 1])
def test_absent_cta_leaves_the_solve_to_the_graph(mp, n, half, absent):
    """Failure detection without a fault: one CTA stays away, the others' wait for
    it runs out after 2 ms and nothing has changed; the solve goes on as a kernel
    per step.  The next one, with all CTAs, is one launch with its usual bits."""
    from drb import _capi as capi
    rp, ci, v = band(n, half)
    a = mp.distributed_sparse_matrix(mp.csr_matrix_view(v, rp, ci, (n, n)), 0)
    rng = np.random.default_rng(n)
    b, x0 = rng.standard_normal(n), rng.standard_normal(n)
    bt = torch.from_numpy(b).cuda()

    def run():
        x = torch.from_numpy(x0.copy()).cuda()
        c0 = capi.launch_count()
        info = mp.conjugate_gradient(a, bt, x, max_iters=9, rtol=0.0)
        assert info["iterations"] == 9
        return x.cpu().numpy(), capi.launch_count() - c0

    usual, launches = run()
    assert launches == 1
    capi.check(capi.lib.drb_csr_cg_set_wait(a.handle, 2_000_000, absent))
    x, launches = run()
    assert launches > 1
    xo = oracle.cg(rp, ci, v, b, x0, 9, 0.0)[0]
    assert np.linalg.norm(x - xo) <= 1e-12 * np.linalg.norm(xo)
    capi.check(capi.lib.drb_csr_cg_set_wait(a.handle, 0, -1))
    again, launches = run()
    assert launches == 1 and np.array_equal(again, usual)

