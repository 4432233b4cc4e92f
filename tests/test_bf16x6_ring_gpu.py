"""BF16x6 128 x 128 tiles whose operands exceed L2 run with a deeper ring and
fewer epilogue warps: the same sums, bit for bit, as pieces of the problem that
fit it, at C widths with whole, partial and odd last chunks."""
import pytest

import cucosma_b200 as cc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("epilogue,beta", [("none", 0.0), ("sigmoid", 0.5)])
@pytest.mark.parametrize("m,n,k", [(100, 9001, 2000), (128, 16000, 1024), (257, 12331, 1100), (1, 64, 300000)])
def test_equals_its_column_blocks(cuda, m, n, k, epilogue, beta):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(m + n)

    def rnd(r, c):
        t = torch.zeros((r, -(-c // 4) * 4), device="cuda")
        t[:, :c] = torch.rand((r, c), generator=g, device="cuda") * 2 - 1
        return t[:, :c]

    A, B, C = rnd(m, k), rnd(k, n), rnd(m, n)
    kw = dict(precision="bf16x6", tile=1, epilogue=epilogue)
    splits = cc.get_plan(cc.make_desc(A, B, C, 1.0, beta, **kw))["splits"]
    whole = rnd(m, n)
    whole.copy_(C)
    cc.gemm(A, B, whole, 1.0, beta, split_k=splits, **kw)
    step = max(4, n // 12 // 4 * 4)
    for c0 in range(0, n, step):
        c1 = min(n, c0 + step)
        part, b = rnd(m, c1 - c0), rnd(k, c1 - c0)
        part.copy_(C[:, c0:c1])
        b.copy_(B[:, c0:c1])
        cc.gemm(A, b, part, 1.0, beta, split_k=splits, **kw)
        assert torch.equal(part, whole[:, c0:c1])
