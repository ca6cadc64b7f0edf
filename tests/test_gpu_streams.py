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
