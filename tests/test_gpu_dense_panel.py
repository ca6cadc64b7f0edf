"""Dense gemv paths against the oracle at the edges of their tiles: the multi-RHS
panel kernel (tiles of 64 or 32 rows in FP32, 64 in FP64; chunks of 64 or 128
columns in FP32, 32 or 64 in FP64; tiles cut between CTAs, aligned and shifted rows,
blocks of at most 32 right-hand sides) and the one-RHS row kernel (rows cut between warps and CTAs)."""
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


def check(mp, dtype, m, n, k, lda, layout, offset=0):
    g = torch.Generator().manual_seed(1000 * m + 10 * n + k)
    buf = torch.full((m * lda + offset,), float("nan"), dtype=dtype)
    A = buf[offset:].view(m, lda)[:, :n]
    A.copy_(torch.randn(m, n, generator=g, dtype=torch.float64))
    X = torch.randn(n, k, generator=g, dtype=torch.float64).to(dtype)
    dev = buf.cuda()
    Ad = dev[offset:].view(m, lda)[:, :n]
    xin = (X.t().contiguous() if layout == 0 else X.contiguous()).cuda()
    y = torch.full((m * k,), float("nan"), dtype=dtype, device="cuda")
    mp.dense_gemv(Ad, xin, y, k, layout)
    y2 = torch.empty_like(y)
    mp.dense_gemv(Ad, xin, y2, k, layout)
    assert torch.equal(y, y2)  # repeatable bit for bit
    Y = (y.cpu().view(k, m).t() if layout == 0 else y.cpu().view(m, k)).double().numpy()
    ref = oracle.dense_gemv(A.double().contiguous().numpy(),
                            X.double().t().contiguous().numpy().ravel(), k,
                            oracle.ACC_LD).reshape(k, m).T
    u = 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -53
    # every output is a sum of n products in some order: at most n roundings each
    bound = (n + 8) * u * (A.double().abs() @ X.double().abs()).numpy()
    assert np.all(np.abs(Y - ref) <= bound)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("m,n,k,lda,layout", [
    (1, 1, 2, 1, 0), (31, 33, 2, 33, 1), (33, 127, 4, 128, 0), (63, 128, 5, 128, 1),
    (64, 129, 8, 132, 0), (65, 31, 9, 31, 1), (127, 32, 12, 32, 0), (128, 640, 13, 643, 0),
    (129, 1000, 16, 1000, 1), (257, 4111, 17, 4111, 0), (300, 2050, 20, 2052, 1),
    (1000, 777, 21, 777, 0), (2000, 515, 24, 516, 1), (95, 6000, 25, 6000, 0),
    (4099, 100, 32, 100, 1), (130, 1500, 33, 1501, 0), (70, 300, 67, 300, 1)])
def test_panel(mp, dtype, m, n, k, lda, layout):
    check(mp, dtype, m, n, k, lda, layout)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("k", [1, 6])
def test_misaligned_base(mp, dtype, k):
    check(mp, dtype, 200, 1024, k, 1024, 0, offset=1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("m,n,lda", [
    (1, 3, 3), (2, 511, 512), (3, 513, 513), (100, 2049, 2052), (889, 1000, 1000),
    (3, 8191, 8192), (5, 8192, 8192), (700, 8201, 8204), (2, 40003, 40004),
    # over 16 MB with few rows per CTA: rows cut between CTAs
    (5, 1_000_003, 1_000_004), (40, 131_073, 131_073), (1500, 3001, 3001),
    # whole rows per CTA
    (5003, 1001, 1001), (9000, 130, 132)])
def test_one_rhs(mp, dtype, m, n, lda):
    check(mp, dtype, m, n, 1, lda, 0)


@pytest.mark.parametrize("dtype,m,n", [
    (torch.float32, 4800, 131_072), (torch.float32, 700, 40_001),  # whole rows per CTA
    (torch.float32, 1, 4_000_000), (torch.float32, 3, 1 << 20), (torch.float32, 2, 700_003),
    (torch.float32, 1, 40_000_000), (torch.float64, 1, 4_000_000), (torch.float64, 3, 700_003)])
def test_one_rhs_sums_do_not_drift(mp, dtype, m, n):
    """Equal products: the additions of one long chain round the same way while
    the sum is in one binade, so a chain's length shows (0.7 in f32, relative:
    4e-5 after 4096 terms, 1.6e-4 after 15600)."""
    A = torch.full((m, n), 0.7, dtype=dtype, device="cuda")
    x = torch.ones(n, dtype=dtype, device="cuda")
    y = torch.empty(m, dtype=dtype, device="cuda")
    mp.dense_gemv(A, x, y, 1, 0)
    u = 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -53
    exact = n * float(A[0, 0])
    # The additions a product passes through: its step's 32, its warp's steps (of 512
    # elements or more; whole rows, or an equal share for two CTAs per SM), a
    # tree of 5, the CTA's 8 warps, a lane's share of 592 CTAs and a tree of 5.
    share = n if m >= 592 else m * n / (2 * 148 * 8) + 512
    bound = (32 + share / 512 + 2 + 5 + 8 + 19 + 5) * u * exact
    assert np.all(np.abs(y.double().cpu().numpy() - exact) <= bound)


def test_nan_stays_in_its_row_and_column(mp):
    A = torch.randn(70, 200, device="cuda")
    x = torch.randn(3 * 200, device="cuda")
    A[5, 7], x[200 + 11] = float("nan"), float("inf")
    y = torch.empty(3 * 70, device="cuda")
    mp.dense_gemv(A, x, y, 3, 0)
    bad = ~torch.isfinite(y.view(3, 70)).cpu()
    want = torch.zeros(3, 70, dtype=torch.bool)
    want[:, 5] = True
    want[1, :] = True
    assert torch.equal(bad, want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("k", [3, 20, 32])
def test_panel_sums_do_not_drift(mp, dtype, k):
    """Equal products, as in test_one_rhs_sums_do_not_drift, in tiles that no
    CTA boundary cuts (more tiles than CTAs)."""
    m, n = 19_000, 16_384
    A = torch.full((m, n), 0.7, dtype=dtype, device="cuda")
    x = torch.ones(n * k, dtype=dtype, device="cuda")
    y = torch.empty(m * k, dtype=dtype, device="cuda")
    mp.dense_gemv(A, x, y, k, 0)
    u = 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -53
    exact = n * float(A[0, 0])
    # The additions a product passes through: 32 until a fold (a lane's in f32, one of
    # two warps' in f64), the folds of the row (512 columns each, or 64), a tree.
    folds = n / 512 if dtype == torch.float32 else n / 64
    bound = (32 + folds + 8) * u * exact
    assert np.all(np.abs(y.double().cpu().numpy() - exact) <= bound)


@pytest.mark.parametrize("dtype,m,n,k,lda,layout", [
    # long chunks (a ring of two): 16-byte rows and shifted ones, both layouts
    (torch.float32, 4100, 4096, 3, 4096, 0), (torch.float32, 4100, 4099, 12, 4099, 1),
    (torch.float32, 4100, 4099, 20, 4100, 0), (torch.float32, 2100, 4099, 25, 4101, 0),
    (torch.float32, 2100, 4096, 32, 4104, 1), (torch.float64, 4097, 4095, 5, 4095, 0),
    (torch.float64, 4097, 4096, 13, 4098, 1), (torch.float64, 4097, 4095, 16, 4097, 0),
    # shares of many tiles, rounded up to whole tiles
    (torch.float32, 310_001, 40, 3, 40, 0), (torch.float32, 155_003, 50, 30, 51, 1),
    (torch.float64, 310_001, 30, 2, 31, 0)])
def test_panel_long_chunks_and_many_tiles(mp, dtype, m, n, k, lda, layout):
    check(mp, dtype, m, n, k, lda, layout)
