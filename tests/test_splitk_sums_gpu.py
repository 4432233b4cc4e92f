"""The split-K reduction's sum over the planes: every remainder of its batches,
with and without the next batch's loads in flight, whole and partial last
vectors of a row.  Whole-number operands make every partial sum exact."""
import pytest

import cucosma_b200 as cc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("beta", [0.0, 2.0])
@pytest.mark.parametrize("splits", [9, 15, 16, 17, 18, 23, 24, 25, 26, 32, 33, 70])
def test_sum_over_splits(cuda, dtype, beta, splits):
    import torch

    dt = getattr(torch, dtype)
    m, n, k = 19, 39, splits * 64
    g = torch.Generator(device="cuda")
    g.manual_seed(splits)

    def ints(r, c):
        t = torch.zeros((r, -(-c // 4) * 4), dtype=dt, device="cuda")
        t[:, :c] = torch.randint(-8, 9, (r, c), generator=g, device="cuda").to(dt)
        return t[:, :c]

    A, B, C = ints(m, k), ints(k, n), ints(m, n)
    want = A.double() @ B.double() + beta * C.double()
    d = cc.make_desc(A, B, C, 1.0, beta, precision="native", split_k=splits)
    plan = cc.get_plan(d)
    assert plan["splits"] == splits
    cc.gemm(A, B, C, 1.0, beta, precision="native", split_k=splits)
    assert torch.equal(C.double(), want)
