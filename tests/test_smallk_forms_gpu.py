"""The small-K kernel with 5 to 8 rows: both its forms (two groups of four rows,
8 rows a thread), K at and between the rows of B loaded at once, ragged ends,
and N long enough that a CTA walks several blocks; guard bands around C."""
import numpy as np
import pytest

import cucosma_b200 as cc
import oracle
from tests._util import check_against_oracle, to_dev, uniform

pytestmark = pytest.mark.gpu

SENTINEL = 321.25
CASES = [(5, 1030, 5), (8, 2051, 16), (6, 513, 13), (7, 1, 1), (5, 400001, 4), (8, 700003, 7), (6, 310007, 3)]


@pytest.mark.parametrize("epilogue,beta", [("none", 0.0), ("sigmoid", 0.0), ("relu", 0.5), ("none", -0.5)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("shape", CASES, ids=["%dx%dx%d" % c for c in CASES])
def test_smallk_vs_oracle(cuda, shape, dtype, epilogue, beta):
    import torch

    m, n, k = shape
    A, B, Cin = uniform(1, (m, k), dtype), uniform(2, (k, n), dtype), uniform(3, (m, n), dtype)
    dA, dB = to_dev(A), to_dev(B)
    ld = -(-n // 4) * 4 + 8
    buf = torch.full((m + 2, ld), SENTINEL, dtype=dA.dtype, device="cuda")
    C = buf[1:1 + m, :n]
    C.copy_(torch.from_numpy(Cin))
    assert cc.get_plan(cc.make_desc(dA, dB, C, 1.25, beta, epilogue=epilogue))["tile_m"] == 8
    cc.gemm(dA, dB, C, 1.25, beta, epilogue=epilogue)
    torch.cuda.synchronize()
    h = buf.cpu().numpy()
    code = {"none": oracle.EPI_NONE, "sigmoid": oracle.EPI_SIGMOID, "relu": oracle.EPI_RELU}[epilogue]
    check_against_oracle(np.ascontiguousarray(h[1:1 + m, :n]), A, B, Cin, 1.25, beta, code, dtype)
    region = np.zeros(h.shape, bool)
    region[1:1 + m, :n] = True
    assert np.all(h[~region] == SENTINEL), "a write landed outside C"
