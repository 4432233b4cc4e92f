"""Split-K inside a cluster (small native launches): parity with the FP64
oracle under the rigorous bound at tile, K and split edges, equal bit for bit
to the workspace reduction of the same split, and inside a stream capture."""
import ctypes as C

import numpy as np
import pytest

import cucosma_b200 as cc
import oracle
from tests._util import check_against_oracle, to_dev, uniform

pytestmark = pytest.mark.gpu

CASES = [(9, 9, 17), (64, 128, 32), (65, 129, 31), (200, 136, 96), (128, 300, 133), (17, 1000, 250)]


@pytest.mark.parametrize("epilogue,beta", [("none", 0.0), ("sigmoid", 0.5)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("split_k", [0, 2, 5, 8])
@pytest.mark.parametrize("shape", CASES, ids=["%dx%dx%d" % c for c in CASES])
def test_cluster_split_vs_oracle(cuda, shape, split_k, dtype, epilogue, beta):
    import torch

    m, n, k = shape
    A, B, Cin = uniform(1, (m, k), dtype), uniform(2, (k, n), dtype), uniform(3, (m, n), dtype)
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(Cin)
    d = cc.make_desc(dA, dB, dC, 1.25, beta, epilogue=epilogue, split_k=split_k)
    plan = cc.get_plan(d)
    ctas = -(-m // plan["tile_m"]) * -(-n // plan["tile_n"]) * plan["splits"]
    clustered = plan["splits"] == 1 or (plan["splits"] <= 8 and ctas <= 80)
    assert (plan["workspace_bytes"] == 0) == clustered and plan["launches"] == (1 if clustered else 2)
    cc.gemm(dA, dB, dC, 1.25, beta, epilogue=epilogue, split_k=split_k)
    torch.cuda.synchronize()
    code = oracle.EPI_SIGMOID if epilogue == "sigmoid" else oracle.EPI_NONE
    check_against_oracle(dC.cpu().numpy(), A, B, Cin, 1.25, beta, code, dtype)


@pytest.mark.parametrize("split_k", [2, 3, 6])
def test_cluster_split_equals_workspace_split(cuda, split_k):
    """The entry point with a fixed scratch array keeps its partial sums there."""
    import torch

    m, n, k = 130, 140, 500
    A, B, Cin = uniform(4, (m, k)), uniform(5, (k, n)), uniform(6, (m, n))
    dA, dB, c1, c2 = to_dev(A), to_dev(B), to_dev(Cin), to_dev(Cin)
    f = cc.lib().cucosma_sgemm_splitk_static
    f.argtypes = [C.c_int] * 3 + [C.c_float, C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_float, C.c_void_p, C.c_int,
                                  C.c_int, C.c_void_p]
    assert f(m, n, k, 1.5, dA.data_ptr(), dA.stride(0), dB.data_ptr(), dB.stride(0), 0.5, c1.data_ptr(), c1.stride(0),
             split_k, torch.cuda.current_stream().cuda_stream) == cc.SUCCESS
    cc.gemm(dA, dB, c2, 1.5, 0.5, split_k=split_k)
    torch.cuda.synchronize()
    assert torch.equal(c1, c2)


def test_cluster_split_in_a_capture(cuda):
    import torch

    A, B = uniform(7, (200, 96)), uniform(8, (96, 136))
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(np.zeros((200, 136), np.float32))
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        cc.cosma_sgemm(dA, dB, dC, stream=s)
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            cc.cosma_sgemm(dA, dB, dC, stream=s)
        dA.mul_(-2.0)
        g.replay()
        s.synchronize()
    check_against_oracle(dC.cpu().numpy(), -2.0 * A, B, None, 1.0, 0.0, oracle.EPI_NONE, np.float32)
