"""The one-launch operand split: the backward pass's planes (G in both
layouts, B's rows, A's columns) at tile and row-unit edges, against the FP64
product of the same FP32 G, and with a workspace that holds one product at a
time."""
import ctypes as C

import numpy as np
import pytest

import cucosma_b200 as cc
from tests._util import bf16_bound, to_dev, uniform

pytestmark = pytest.mark.gpu

# the smallest; one past / short of a 64 x 64 tile and of an 8-column group; a row longer than one 2048-column unit
SHAPES = [(1, 1, 1), (65, 63, 64), (130, 70, 45), (64, 128, 9), (40, 2051, 33), (2049, 31, 130)]


@pytest.mark.parametrize("epilogue", ["none", "sigmoid", "relu"])
@pytest.mark.parametrize("precision,nterms", [("bf16x3", 2), ("bf16x6", 3)])
@pytest.mark.parametrize("shape", SHAPES, ids=["%dx%dx%d" % s for s in SHAPES])
def test_backward_planes_at_edges(cuda, shape, precision, nterms, epilogue):
    import torch

    m, n, k = shape
    A, B, dY = uniform(1, (m, k)), uniform(2, (k, n)), uniform(3, (m, n))
    Y = uniform(4, (m, n), lo=0.0 if epilogue == "sigmoid" else -1.0)
    alpha = np.float32(0.75)
    G = alpha * dY
    if epilogue == "sigmoid":
        G = G * (Y * (np.float32(1) - Y))
    elif epilogue == "relu":
        G = np.where(Y > 0, G, np.float32(0))
    tA, tB, tY, tdY = to_dev(A), to_dev(B), to_dev(Y), to_dev(dY)
    out = []
    d = cc.make_desc(tA, tB, tY, float(alpha), 0.0, precision=precision, epilogue=epilogue)
    need = C.c_size_t(0)
    assert cc.lib().cucosma_gemm_backward_workspace_size(C.byref(d), C.byref(need)) == cc.SUCCESS
    # the larger product's own part: what the two products need when they share it (the flag's plan is the
    # backward pass's: never the fused split, whose workspace holds no planes)
    parts = []
    for pm, pn, pk in ((m, k, n), (k, n, m)):
        a, b, c = (torch.empty(r, -(-q // 4) * 4, device="cuda")[:, :q] for r, q in ((pm, pk), (pk, pn), (pm, pn)))
        parts.append(cc.workspace_size(cc.make_desc(a, b, c, precision=precision, flags=cc.FLAG_TEST_SKIP_STAGE)))
    assert need.value >= max(parts)
    for size in (need.value, max(parts)):
        dA, dB = to_dev(np.zeros_like(A)), to_dev(np.zeros_like(B))
        ws = torch.empty(max(size, 256), dtype=torch.uint8, device="cuda")
        cc.gemm_backward(tA, tB, tY, tdY, dA, dB, alpha=float(alpha), precision=precision, epilogue=epilogue, workspace=ws)
        torch.cuda.synchronize()
        out.append((dA.cpu().numpy(), dB.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    for got, P, Q in ((out[0][0], G, np.ascontiguousarray(B.T)), (out[0][1], np.ascontiguousarray(A.T), G)):
        ref, b = bf16_bound(P, Q, None, 1.0, 0.0, nterms)
        assert np.all(np.abs(got - ref) <= b)
    assert cc.device_status() == (cc.SUCCESS, 0)
