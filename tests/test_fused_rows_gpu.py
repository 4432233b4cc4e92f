"""The fused-split kernels on a C that is read and whose rows end off the
16-byte boundary (long K, so that C is the lesser traffic): beta * C joins the
accumulators with one rounding, edge tiles and guard bands included."""
import pytest

import cucosma_b200 as cc

pytestmark = pytest.mark.gpu

SENTINEL = 77.5
SHAPES = [(300, 131, 8200), (257, 1, 5000), (200, 258, 9000), (512, 1023, 4096), (700, 66, 4097)]


@pytest.mark.parametrize("epilogue", ["none", "relu", "sigmoid"])
@pytest.mark.parametrize("precision,tile", [("bf16x3", 5), ("bf16x6", 4)])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_c_by_rows(cuda, m, n, k, precision, tile, epilogue):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(8)

    def mat(r, c, pad=0):
        t = torch.full((r + pad, -(-c // 4) * 4 + 2 * pad), SENTINEL, device="cuda")
        t[pad // 2:pad // 2 + r, :c] = torch.rand((r, c), generator=g, device="cuda") * 2 - 1
        return t, t[pad // 2:pad // 2 + r, :c]

    (_, A), (_, B), (buf, C), (_, P) = mat(m, k), mat(k, n), mat(m, n, 4), mat(m, n)
    kw = dict(precision=precision, tile=tile, split_k=1)
    assert cc.get_plan(cc.make_desc(A, B, C, 1.0, 0.5, **kw))["fused"] == 1
    before = buf.clone()
    cc.gemm(A, B, P, 1.0, 0.0, **kw)
    cc.gemm(A, B, C, 1.0, 0.5, epilogue=epilogue, **kw)
    z = (before[2:2 + m, :n].double() * 0.5 + P.double()).float()  # exact in 64 bits, rounded once
    if epilogue == "sigmoid":
        # within a few ulp of the sigmoid of z
        assert float((C.double() - torch.sigmoid(z.double())).abs().max()) <= 8 * 2.0 ** -24
    else:
        assert torch.equal(C, z.clamp_min(0) if epilogue == "relu" else z)
    after = buf.clone()
    after[2:2 + m, :n] = before[2:2 + m, :n]
    assert torch.equal(after, before), "a write landed outside C"
    assert cc.device_status() == (cc.SUCCESS, 0)
