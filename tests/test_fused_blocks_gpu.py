"""Fused BF16 tiles with C heavy: one or two staging blocks by the epilogue and
the length of K.  The results equal those of the pre-pass path bit for bit on
both sides of every line, at widths with no, a partial and a partial second
last chunk of 32 columns."""
import pytest

import cucosma_b200 as cc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,ftile,utile", [("bf16x3", 5, 4), ("bf16x6", 4, 2)])
@pytest.mark.parametrize("epilogue,beta", [("none", 0.0), ("relu", 0.5), ("sigmoid", 0.0), ("sigmoid", 0.5)])
@pytest.mark.parametrize("n", [128, 200, 236, 331])
@pytest.mark.parametrize("k", [40, 96, 104, 130, 160, 163, 256, 260, 449, 641])
def test_equals_the_prepass_path(cuda, precision, ftile, utile, epilogue, beta, n, k):
    import torch

    m = 3001
    g = torch.Generator(device="cuda")
    g.manual_seed(n * k)

    def rnd(r, c):
        t = torch.zeros((r, -(-c // 4) * 4), device="cuda")
        t[:, :c] = torch.rand((r, c), generator=g, device="cuda") * 2 - 1
        return t[:, :c]

    A, B, C = rnd(m, k), rnd(k, n), rnd(m, n)
    D = rnd(m, n)
    D.copy_(C)
    kw = dict(precision=precision, epilogue=epilogue, split_k=1)
    assert cc.get_plan(cc.make_desc(A, B, C, 1.0, beta, tile=ftile, **kw))["fused"] == 1
    cc.gemm(A, B, C, 1.0, beta, tile=ftile, **kw)
    cc.gemm(A, B, D, 1.0, beta, tile=utile, **kw)
    assert torch.equal(C, D)
