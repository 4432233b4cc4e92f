"""BF16 paths whose whole K is one accumulator chunk (K <= 256): the epilogue
reads the tile from TMEM block by block.  Checked against the FP64 oracle at
the edges of its 64-column blocks, 32-column chunks and 256-row tiles, with
enough tiles that a CTA pair walks several, and with guard bands around C."""
import numpy as np
import pytest

import cucosma_b200 as cc
import oracle
from tests._util import bf16_bound, to_dev, uniform

pytestmark = pytest.mark.gpu

SENTINEL = 1234.5
# (m, n, k): the smallest; one column short of and past a chunk and a block; a
# quarter granule; the last short K; several tiles a pair in N, and in M
SHAPES = [(129, 1, 1), (130, 31, 7), (256, 33, 32), (257, 95, 256), (300, 65, 255), (200, 130, 64), (513, 259, 96),
          (129, 20515, 33), (20500, 70, 40)]
# the pair tile and the fused-split tile of BF16x3, the fused tile of BF16x6
TILES = [("bf16x3", 2, 4), ("bf16x3", 2, 5), ("bf16x6", 3, 4)]


@pytest.mark.parametrize("epilogue,beta", [("none", 0.5), ("sigmoid", 0.5), ("relu", 0.0)])
@pytest.mark.parametrize("precision,nterms,tile", TILES, ids=["%s-t%d" % (t[0], t[2]) for t in TILES])
@pytest.mark.parametrize("shape", SHAPES, ids=["%dx%dx%d" % s for s in SHAPES])
def test_short_k_vs_oracle(cuda, shape, precision, nterms, tile, epilogue, beta):
    import torch

    m, n, k = shape
    A, B, Cin = uniform(1, (m, k)), uniform(2, (k, n)), uniform(3, (m, n))
    dA, dB = to_dev(A), to_dev(B)
    ld = -(-n // 4) * 4 + 8
    buf = torch.full((m + 4, ld), SENTINEL, dtype=torch.float32, device="cuda")
    C = buf[2:2 + m, :n]
    C.copy_(torch.from_numpy(Cin))
    cc.gemm(dA, dB, C, 1.0, beta, precision=precision, epilogue=epilogue, tile=tile)
    torch.cuda.synchronize()
    h = buf.cpu().numpy()
    out = h[2:2 + m, :n].astype(np.float64)
    # the activation is 1-Lipschitz (the sigmoid 1/4) and rounds within a few ulp
    _, b = bf16_bound(A, B, Cin, 1.0, beta, nterms)
    ref = oracle.gemm(A, B, Cin, 1.0, beta, {"none": oracle.EPI_NONE, "sigmoid": oracle.EPI_SIGMOID,
                                             "relu": oracle.EPI_RELU}[epilogue])
    assert np.all(np.abs(out - ref) <= (0.25 if epilogue == "sigmoid" else 1.0) * b + 8 * 2.0 ** -24)
    region = np.zeros(h.shape, bool)
    region[2:2 + m, :n] = True
    assert np.all(h[~region] == SENTINEL), "a write landed outside C"
    assert cc.device_status() == (cc.SUCCESS, 0)
