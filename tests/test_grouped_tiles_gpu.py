"""Grouped launches: the tiles the automatic choice takes equal the 128 x 128
tile bit for bit, on batches whose work list has empty positions, one unit,
rows longer than one pre-pass unit and column strips of several tiles."""
import pytest

import cucosma_b200 as cc

pytestmark = pytest.mark.gpu

BATCHES = {
    "one": [(1, 1, 1)],
    "edges": [(129, 257, 33), (256, 128, 320), (257, 129, 65), (64, 2000, 31), (1, 300, 4099), (31, 65, 2113)],
    # more than two waves of 128 x 128 tiles: the automatic choice may take a pair tile
    "waves": [(2048, 1500, 200), (1000, 2048, 777), (700, 1100, 1300), (2040, 260, 64), (130, 1999, 2300)],
}


@pytest.mark.parametrize("precision,tiles", [("bf16x3", (0, 4, 5)), ("bf16x6", (0, 2))])
@pytest.mark.parametrize("batch", list(BATCHES))
def test_grouped_tiles_bit_identical(cuda, batch, precision, tiles):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(11)

    def mat(r, c):
        return (torch.rand((r, -(-c // 4) * 4), generator=g, device="cuda") * 2 - 1)[:, :c]

    ops = [(mat(m, k), mat(k, n), mat(m, n)) for m, n, k in BATCHES[batch]]

    def run(tile):
        probs = [(A, B, C._base.clone()[:, :C.shape[1]]) for A, B, C in ops]  # (keeps the padded rows)
        cc.grouped(probs, precision=precision, alpha=1.25, beta=0.5, tile=tile)()
        torch.cuda.synchronize()
        return [p[2] for p in probs]

    want = run(1)
    for tile in tiles:
        for got, ref in zip(run(tile), want):
            assert torch.equal(got, ref), tile
    assert cc.device_status() == (cc.SUCCESS, 0)
