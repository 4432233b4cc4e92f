"""cucosma_tune where the automatic BF16 plan is not one of the tile ids and
split counts: its K-split last wave is a candidate, and fused tiles are where
the plan takes them."""
import pytest

import cucosma_b200 as cc

pytestmark = pytest.mark.gpu


def operands(torch, m, n, k):
    g = torch.Generator(device="cuda")
    g.manual_seed(2)

    def mat(r, c):
        return (torch.rand((r, -(-c // 4) * 4), generator=g, device="cuda") * 2 - 1)[:, :c]

    return mat(m, k), mat(k, n), mat(m, n)


@pytest.mark.parametrize("precision", ["bf16x3", "bf16x6"])
def test_k_split_last_wave_is_a_candidate(cuda, precision, tmp_path):
    import torch

    cc.tune_cache_clear()
    try:
        A, B, C = operands(torch, 2300, 4345, 5000)
        d = cc.make_desc(A, B, C, precision=precision)
        untuned = cc.get_plan(d)
        assert untuned["launches"] == 3 and untuned["splits"] == 1  # its last wave is split
        for _ in range(2):  # a second time past the first's cache entry
            r = cc.tune(A, B, C, precision=precision, max_candidates=1)
            assert (r["split_k"], r["swizzle"], r["tile"], r["candidates"]) == (0, 0, 0, 1) and r["ms"] > 0
            assert cc.get_plan(d) == untuned
        path = str(tmp_path / "cache.txt")
        cc.tune_cache_save(path)
        cc.tune_cache_clear()
        cc.tune_cache_load(path)
        assert cc.tune_cache_size() == 1 and cc.get_plan(d) == untuned
        # an entry of another configuration does not stand in for the library's choice
        cc.tune_cache_clear()
        with open(path) as f:
            line = f.read().split()
        line[8:11] = ["1", "8", "2" if precision == "bf16x3" else "1"]
        with open(path, "w") as f:
            f.write(" ".join(line) + "\n")
        cc.tune_cache_load(path)
        assert cc.get_plan(d) != untuned
        assert cc.tune(A, B, C, precision=precision, max_candidates=1)["tile"] == 0
        assert cc.get_plan(d) == untuned
    finally:
        cc.tune_cache_clear()


@pytest.mark.parametrize("precision,tile", [("bf16x3", 5), ("bf16x6", 4)])
def test_fused_tile_is_a_candidate_where_the_plan_takes_it(cuda, precision, tile):
    import torch

    cc.tune_cache_clear()
    try:
        A, B, C = operands(torch, 256, 8192, 256)
        assert cc.get_plan(cc.make_desc(A, B, C, precision=precision))["fused"] == 1
        few = cc.tune(A, B, C, precision=precision)
        per_tile = cc.tune(A, B, C, precision=precision, max_candidates=1)["candidates"]
        assert per_tile == 1 and few["candidates"] % 4 == 0  # four tiles of as many bands and splits each
    finally:
        cc.tune_cache_clear()


@pytest.mark.parametrize("m,n,k", [(200, 300, 500), (3000, 2900, 200)])
def test_occupancy_of_the_fp64_tile(cuda, m, n, k):
    """Four 64 x 64 CTAs an SM, one of 128 x 128."""
    import torch

    cc.tune_cache_clear()
    try:
        A, B, C = (t.double() for t in operands(torch, m, n, k))
        A, B, C = (torch.zeros((t.shape[0], t.shape[1] + t.shape[1] % 2), dtype=t.dtype, device="cuda")[:, :t.shape[1]]
                   .copy_(t) for t in (A, B, C))
        r = cc.tune(A, B, C)
        tile_m = cc.get_plan(cc.make_desc(A, B, C))["tile_m"]
        assert r["occupancy"] == (4 if tile_m == 64 else 1)
    finally:
        cc.tune_cache_clear()
