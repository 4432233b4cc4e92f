"""The native FP64 call's K splits: no output is a longer chain of roundings
than 128 x 128 tiles summed through the workspace give, whatever tile or
reduction the plan takes.  Integer operands below 2^26 make the exact result
available, so the rounding errors of the two can be compared."""
import numpy as np
import pytest

import cucosma_b200 as cc

pytestmark = pytest.mark.gpu

# (m, n, k) and the K splits of the fastest 128 x 128 plan of 148 SMs
CASES = [((800, 600, 1200), 4), ((500, 500, 500), 8), ((1000, 777, 1531), 5), ((2000, 2000, 2000), 4),
         ((195, 655, 1710), 12), ((264, 157, 703), 11), ((357, 1191, 145), 2), ((768, 360, 256), 4),
         ((334, 434, 125), 2), ((3000, 3000, 3000), 1)]


@pytest.mark.parametrize("shape,splits", CASES, ids=["%dx%dx%d" % c[0] for c in CASES])
def test_rounding_error_of_the_chosen_plan(cuda, shape, splits):
    import torch

    m, n, k = shape
    g = torch.Generator(device="cuda")
    g.manual_seed(9)

    def ints(r, c):
        t = torch.zeros((r, c + c % 2), dtype=torch.float64, device="cuda")
        t[:, :c] = torch.randint(-2**26, 2**26, (r, c), generator=g, device="cuda").double()
        return t[:, :c]

    A, B = ints(m, k), ints(k, n)
    # A = 2^13 hi + lo: both products are integers below 2^53, exact in 64 bits
    hi = torch.round(A / 8192)
    ph, pl = (hi @ B) * 8192.0, (A - 8192.0 * hi) @ B

    def rms(**kw):
        C = torch.zeros((m, n + n % 2), dtype=torch.float64, device="cuda")[:, :n]
        cc.gemm(A, B, C, **kw)
        return float(((C - ph) - pl).pow(2).mean().sqrt())

    plan = cc.get_plan(cc.make_desc(A, B, A.new_zeros((m, n + n % 2))[:, :n]))
    kchunk = -(-(-(-k // splits)) // 16) * 16
    assert plan["kchunk"] <= kchunk
    # shorter chains cannot err more; equal ones give the same bits.  The
    # sample of m * n errors says so to 4 / sqrt(2 m n).
    assert rms() <= rms(tile=1, split_k=splits) * (1 + 4 / np.sqrt(2 * m * n))


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("m", [65535 * 64, 65535 * 64 + 1])
def test_most_tile_rows_of_a_grid(cuda, dtype, m):
    """64-row tiles only while their count fits one grid dimension; sampled rows of a tall, narrow C."""
    import torch

    dt = getattr(torch, dtype)
    n, k = 12, 20
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    A = torch.randint(-8, 9, (m, k), generator=g, device="cuda").to(dt)
    B = torch.randint(-8, 9, (k, n), generator=g, device="cuda").to(dt)
    C = torch.full((m, n), -1.0, dtype=dt, device="cuda")
    assert -(-m // cc.get_plan(cc.make_desc(A, B, C))["tile_m"]) <= 65535
    cc.gemm(A, B, C)
    assert torch.equal(C, A @ B)  # small integers: exact in any order
