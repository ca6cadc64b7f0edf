"""The dense BF16 batch where its work is cut differently: few tiles (cut along K
into parts that a second kernel adds), X read in place (columns on 16 bytes) or
packed (odd sizes, row-major), one or several matrices in one plan."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

COL, ROW = 0, 1


@pytest.fixture(scope="module")
def mp():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from drb import mp as _mp
    return _mp


@pytest.mark.parametrize("shapes,k,layout,variant", [
    ([(1, 1)], 1, COL, 1), ([(128, 1024)], 32, COL, 1), ([(129, 1023)], 32, COL, 1),
    ([(700, 4100)], 16, ROW, 1), ([(300, 8192)], 3, COL, 3), ([(257, 5000)], 40, COL, 4),
    ([(1000, 2056), (64, 600), (33, 64)], 20, COL, 0), ([(513, 6001), (2, 9000)], 128, ROW, 2),
    ([(100, 16000)], 200, COL, 1), ([(130, 640)] * 200, 8, COL, 1)])
def test_units(mp, shapes, k, layout, variant):
    if variant == 2 and k > 100:
        variant = 0  # the eight-stage ring does not fit this many right-hand sides
    g = torch.Generator(device="cuda").manual_seed(len(shapes) * 1000 + k)
    As, xs, xcs, ys = [], [], [], []
    for m, n in shapes:
        lda = (n + 7) // 8 * 8
        A = torch.randn(m, lda, device="cuda", generator=g).bfloat16()
        if lda > n:
            A[:, n:] = float("nan")  # padding is never used
        xc = torch.randn(n * k, device="cuda", generator=g).bfloat16()
        As.append(A[:, :n])
        xcs.append(xc)
        xs.append(xc if layout == COL else xc.view(k, n).t().contiguous().view(-1))
        ys.append(torch.full((m * k,), float("nan"), device="cuda"))
    P = mp.dense_batch(As, xs, ys, k, layout)
    P.set_variant(variant)
    P.gemv()
    P.check()
    first = [y.clone() for y in ys]
    for y in ys:
        y.fill_(float("nan"))
    P.gemv()
    P.check()
    for (m, n), A, xc, y, y1 in list(zip(shapes, As, xcs, ys, first))[:4]:
        assert torch.equal(y, y1)
        got = (y.view(m, k).t().reshape(-1) if layout == ROW else y).cpu().double().numpy()
        a, xv = A.double().cpu().numpy(), xc.double().cpu().numpy()
        ref = oracle.dense_gemv(np.ascontiguousarray(a), xv, k, oracle.ACC_F64)
        den = oracle.dense_gemv(np.ascontiguousarray(np.abs(a)), np.abs(xv), k, oracle.ACC_F64)
        # exact products; every accumulation step rounds (or truncates) once: 2^-23
        assert np.all(np.abs(got - ref) <= (n + 8) * 2.0 ** -23 * den)
    P.destroy()


@pytest.mark.parametrize("shapes,k,layout", [
    ([(100, 16000)], 200, COL), ([(513, 6001), (2, 9000)], 128, ROW), ([(300, 8192)], 3, COL),
    ([(257, 5000)], 40, ROW), ([(129, 1023)], 32, COL), ([(128, 1088)], 32, COL)])
def test_every_column_counts_once(mp, shapes, k, layout):
    """Small integers: every sum is exact in FP32, so a column that a cut along K
    drops or takes twice shows."""
    g = torch.Generator(device="cuda").manual_seed(k)
    As, xs, ys, want = [], [], [], []
    for m, n in shapes:
        lda = (n + 7) // 8 * 8
        A = torch.randint(-8, 9, (m, lda), device="cuda", generator=g).bfloat16()
        if lda > n:
            A[:, n:] = float("nan")
        X = torch.randint(-8, 9, (k, n), device="cuda", generator=g).bfloat16()
        assert n * 64 < 2 ** 24
        As.append(A[:, :n])
        xs.append((X if layout == COL else X.t()).contiguous().view(-1))
        ys.append(torch.full((m * k,), float("nan"), device="cuda"))
        want.append((A[:, :n].double() @ X.double().t()).float())
    P = mp.dense_batch(As, xs, ys, k, layout)
    P.gemv()
    P.check()
    for (m, _), y, w in zip(shapes, ys, want):
        assert torch.equal(y.view(m, k) if layout == ROW else y.view(k, m).t(), w)
    P.destroy()
