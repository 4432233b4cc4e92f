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


@pytest.mark.parametrize("precision,utile", [("bf16x3", 4), ("bf16x6", 2)])
@pytest.mark.parametrize("m,n,k,fused", [(72739, 200, 161, 1), (30011, 1000, 384, None), (8193, 2052, 96, None),
                                         (8200, 132, 384, None), (60001, 331, 100, None)])
def test_tall_calls_of_short_k(cuda, precision, utile, m, n, k, fused):
    """Automatic calls with a tall C beyond L2 are fused; any plan's result
    equals the pre-pass path's, bit for bit."""
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    A = torch.zeros((m, -(-k // 4) * 4), device="cuda")[:, :k]
    A.copy_(torch.rand((m, k), generator=g, device="cuda") * 2 - 1)
    B, C, D = (torch.zeros((r, -(-n // 4) * 4), device="cuda")[:, :n] for r in (k, m, m))
    B.copy_(torch.rand((k, n), generator=g, device="cuda") * 2 - 1)
    plan = cc.get_plan(cc.make_desc(A, B, C, precision=precision))
    assert fused is None or plan["fused"] == fused
    cc.gemm(A, B, C, precision=precision)
    if plan["fused"]:
        cc.gemm(A, B, D, precision=precision, tile=utile, split_k=plan["splits"])
        assert torch.equal(C, D)
    else:
        ref = A.double() @ B.double()
        err = (C - ref).abs().amax() / (A.abs().double() @ B.abs().double()).amax()
        assert float(err) <= 2.0 ** (-15 if precision == "bf16x3" else -21)
