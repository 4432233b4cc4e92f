"""cucosma_tune_grouped beside plans with the automatic tile."""
import pytest

import cucosma_b200 as cc

pytestmark = pytest.mark.gpu

# more than two waves of 128 x 128 tiles, where the automatic tile is a pair tile
WAVES = [(2048, 1500, 200), (1000, 2048, 777), (700, 1100, 1300), (2040, 260, 64), (130, 1999, 2300)]


def problems(torch, shapes, seed=3):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def mat(r, c):
        return (torch.rand((r, -(-c // 4) * 4), generator=g, device="cuda") * 2 - 1)[:, :c]

    return [(mat(m, k), mat(k, n), mat(m, n)) for m, n, k in shapes]


@pytest.mark.parametrize("precision,tile", [("bf16x3", 0), ("bf16x3", 1), ("bf16x3", 3), ("bf16x6", 0), ("bf16x6", 1)])
def test_plan_outlives_a_tune_on_its_workspace(cuda, precision, tile):
    import torch

    cc.tune_cache_clear()
    try:
        probs = problems(torch, WAVES)
        plan = cc.grouped(probs, precision=precision, tile=tile)
        kept = plan.tile()
        plan()
        torch.cuda.synchronize()
        want = [p[2].clone() for p in probs]
        before = plan.workspace.clone()
        plan.tune()
        # the plan's tables are byte for byte those it was made with, so it can
        # be launched again: problem records, block starts, work list (whole
        # rounds of one unit a CTA or pair), each from a 256-byte boundary;
        # a launch reads nothing else of the workspace that it has not written
        _, tm, tn, _ = kept
        units = sum(-(-m // tm) * -(-n // tn) for m, n, _ in WAVES)
        slots = [min(units, s) for s in ([148] if tm == 128 else range(64, 75))]
        n = len(WAVES)
        tables = sum(-(-b // 256) * 256 for b in (384 * n, 16 * n)) + 8 * min(-(-units // s) * s for s in slots)
        assert torch.equal(plan.workspace[:tables], before[:tables])
        for p in probs:
            p[2].zero_()
        plan()
        torch.cuda.synchronize()
        assert plan.tile() == kept
        for p, w in zip(probs, want):
            assert torch.equal(p[2], w)
        assert cc.device_status() == (cc.SUCCESS, 0)
    finally:
        cc.tune_cache_clear()


@pytest.mark.parametrize("precision,candidates", [("bf16x3", 4), ("bf16x6", 2)])
def test_tune_measures_the_automatic_tile(cuda, precision, candidates):
    """A batch whose automatic tile (BF16x3) is not 128 x 128: every tile fits the
    plan's workspace, and the automatic one is measured with the others."""
    import torch

    cc.tune_cache_clear()
    try:
        probs = problems(torch, WAVES)
        plan = cc.grouped(probs, precision=precision)
        automatic = plan.tile()[0]
        assert automatic != 1 or precision == "bf16x6"
        r = plan.tune()
        assert r["candidates"] == candidates and r["tile"] in {1, 2, 3, automatic}
        tuned = cc.grouped(probs, precision=precision)
        assert tuned.tile()[0] == r["tile"] and tuned.tile()[3]
        assert tuned.workspace.numel() == plan.workspace.numel()
    finally:
        cc.tune_cache_clear()
