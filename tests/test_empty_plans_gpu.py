"""Plan and workspace queries of problems with an empty dimension answer; they
divided by the number of tiles or K blocks."""
import pytest

import cucosma_b200 as cc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["native", "bf16x3", "bf16x6", "ozaki"])
@pytest.mark.parametrize("m,n,k", [(0, 64, 64), (64, 0, 64), (64, 64, 0), (0, 0, 0), (300, 0, 5000)])
def test_query_answers(cuda, precision, m, n, k):
    import torch

    dt = torch.float64 if precision == "ozaki" else torch.float32
    d = cc.make_desc(*(torch.empty(s, dtype=dt, device="cuda") for s in ((64, 64), (64, 64), (64, 64))),
                     precision=precision)
    d.m, d.n, d.k = m, n, k
    plan = cc.get_plan(d)
    assert plan["splits"] >= 1 and plan["tile_m"] > 0 and plan["tile_n"] > 0
    assert cc.workspace_size(d) == 0
