"""Grouped workspace queries at their limits (no GPU: validation and sizes only):
batches of very many tiles are answered without walking them, more tiles than
their numbers hold and unknown tile ids are refused."""
import ctypes as C
import time

import pytest

import cucosma_b200 as cc


def query(problems, precision="bf16x3", tile=0):
    d = cc.GemmDesc()
    cc.lib().cucosma_gemm_desc_init(C.byref(d))
    d.precision, d.tile = cc.PRECISIONS[precision], tile
    d.dtype = 1 if precision == "ozaki" else 0
    arr = (cc._ext.Problem * len(problems))()
    for i, (m, n, k) in enumerate(problems):
        arr[i] = cc._ext.Problem(m, n, k, -(-k // 4) * 4, -(-n // 4) * 4, -(-n // 4) * 4, 0x10000, 0x10000, 0x10000)
    size = C.c_size_t(0)
    t = time.process_time()
    s = cc.lib().cucosma_grouped_workspace_size(C.byref(d), arr, len(problems), C.byref(size))
    return s, size.value, time.process_time() - t


@pytest.mark.parametrize("precision,terms", [("bf16x3", 2), ("bf16x6", 3)])
def test_many_tiles_are_answered_at_once(precision, terms):
    # 31250 x 31250 tiles of 128 x 128; planes of terms * 2 bytes a value
    s, size, seconds = query([(4000000, 4000000, 8), (100, 100, 100)], precision)
    assert s == cc.SUCCESS and size >= 2 * 4000000 * 8 * 2 * terms
    # dealing 10^9 tiles out takes minutes; some 10^6 at most are dealt out (0.1 s here)
    assert seconds < 5


@pytest.mark.parametrize("precision", ["bf16x3", "bf16x6", "ozaki"])
def test_more_tiles_than_their_numbers_hold(precision):
    big = 2**31 - 1
    for probs in ([(big, big, 8)], [(6000000, 6000000, 8)], [(8, big, 8)] * 200):
        s, _, seconds = query(probs, precision)
        assert s == cc.NOT_SUPPORTED and seconds < 5
    assert query([(6000000, 4000, 8)], precision)[0] == cc.SUCCESS


@pytest.mark.parametrize("precision,ids", [("bf16x3", 5), ("bf16x6", 2), ("ozaki", 1)])
def test_tile_ids(precision, ids):
    for tile in range(-2, 8):
        ok = 0 <= tile <= ids
        assert query([(300, 200, 100)], precision, tile)[0] == (cc.SUCCESS if ok else cc.NOT_SUPPORTED), tile


@pytest.mark.parametrize("precision,ids", [("bf16x3", 5), ("bf16x6", 2), ("ozaki", 1)])
def test_size_asked_for_with_tile_0_holds_every_tile(precision, ids):
    waves = [(2048, 1500, 200), (1000, 2048, 777), (700, 1100, 1300), (2040, 260, 64), (130, 1999, 2300)]
    for probs in (waves, waves * 20, [(10, 10, 10)], [(900, 1, 30)] * 700):
        any_tile = query(probs, precision)[1]
        assert any_tile == max(query(probs, precision, tile)[1] for tile in range(1, ids + 1))
