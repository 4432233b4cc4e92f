"""The thin kernel's block forms (4 or 8 rows, 4 or 8 columns) at their edges,
with K short of, at and past the k-steps a CTA loads at once, one and many
splits, against the FP64 oracle under the rigorous bound."""
import numpy as np
import pytest

import cucosma_b200 as cc
import oracle
from tests._util import check_against_oracle, to_dev, uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("k,split_k", [(17, 0), (255, 1), (1025, 1), (2309, 0), (70001, 0), (9000, 7)])
@pytest.mark.parametrize("m,n", [(1, 1), (4, 4), (4, 5), (5, 4), (8, 8), (3, 9), (12, 7), (1, 13)])
def test_thin_blocks_vs_oracle(cuda, m, n, k, split_k, dtype):
    import torch

    A, B, Cin = uniform(1, (m, k), dtype), uniform(2, (k, n), dtype), uniform(3, (m, n), dtype)
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(Cin)
    cc.gemm(dA, dB, dC, 1.25, -0.5, split_k=split_k)
    torch.cuda.synchronize()
    check_against_oracle(dC.cpu().numpy(), A, B, Cin, 1.25, -0.5, oracle.EPI_NONE, dtype)
