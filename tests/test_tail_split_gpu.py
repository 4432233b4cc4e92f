"""BF16 calls whose last wave of 256 x 256 pair tiles is split along K and
reduced by a second kernel: sampled rows (every tile's edges among them)
against the FP64 oracle, with guard bands around C and a repeated run."""
import numpy as np
import pytest

import cucosma_b200 as cc
import oracle
from tests._util import bf16_bound, to_dev, uniform

pytestmark = pytest.mark.gpu

SENTINEL = 1234.5
# more tiles than pairs, operands larger than L2; ragged in every direction, N
# with a last chunk of less than 32 columns and of less than 4.  The first two
# leave 5 to 9 and 9 to 15 tiles for the last wave of 72 to 74 pairs and are
# always split; the others leave up to 50, where the plan decides.
SPLIT = [(2300, 4345, 5000), (5300, 2801, 4103)]
SHAPES = SPLIT + [(4100, 4090, 4096), (8200, 8101, 2053)]


@pytest.mark.parametrize("epilogue,beta", [("none", 0.0), ("sigmoid", 0.5)])
@pytest.mark.parametrize("precision,nterms", [("bf16x3", 2), ("bf16x6", 3)])
@pytest.mark.parametrize("shape", SHAPES, ids=["%dx%dx%d" % s for s in SHAPES])
def test_tail_split_vs_oracle(cuda, shape, precision, nterms, epilogue, beta):
    import torch

    m, n, k = shape
    A, B, Cin = uniform(1, (m, k)), uniform(2, (k, n)), uniform(3, (m, n))
    dA, dB = to_dev(A), to_dev(B)
    ld = -(-n // 4) * 4 + 8
    runs = []
    for _ in range(2):
        buf = torch.full((m + 4, ld), SENTINEL, dtype=torch.float32, device="cuda")
        C = buf[2:2 + m, :n]
        C.copy_(torch.from_numpy(Cin))
        plan = cc.get_plan(cc.make_desc(dA, dB, C, 1.0, beta, precision=precision, epilogue=epilogue))
        assert (plan["tile_m"], plan["tile_n"], plan["splits"]) == (256, 256, 1)
        assert plan["launches"] == 3 or shape not in SPLIT
        cc.gemm(dA, dB, C, 1.0, beta, precision=precision, epilogue=epilogue)
        torch.cuda.synchronize()
        runs.append(buf.cpu().numpy())
    assert np.array_equal(runs[0], runs[1])
    h = runs[0]
    rows = np.unique(np.r_[np.arange(0, m, 256), np.arange(255, m, 256), np.arange(97, m, 509), m - 1])
    _, b = bf16_bound(A[rows], B, Cin[rows], 1.0, beta, nterms)
    ref = oracle.gemm(A[rows], B, Cin[rows], 1.0, beta,
                      oracle.EPI_SIGMOID if epilogue == "sigmoid" else oracle.EPI_NONE)
    # the sigmoid is 1/4-Lipschitz and rounds within a few ulp
    out = h[2 + rows, :n].astype(np.float64)
    assert np.all(np.abs(out - ref) <= (0.25 if epilogue == "sigmoid" else 1.0) * b + 8 * 2.0 ** -24)
    region = np.zeros(h.shape, bool)
    region[2:2 + m, :n] = True
    assert np.all(h[~region] == SENTINEL), "a write landed outside C"
    assert cc.device_status() == (cc.SUCCESS, 0)
