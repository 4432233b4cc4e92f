"""Grouped launches of many small problems: counts at and around the pre-pass
blocks' search steps (256, 65536), with larger problems of several pre-pass
blocks among them, against batched products in 64 bits."""
import pytest

import cucosma_b200 as cc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["bf16x3", "ozaki"])
@pytest.mark.parametrize("count", [1, 2, 255, 256, 257, 513, 65536, 65537])
def test_counts(cuda, count, precision):
    import torch

    dt = torch.float64 if precision == "ozaki" else torch.float32
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    # 8 x 8 x 8 problems, every 97th (and the last) 72 x 136 x 40; integers, so every form is exact
    big = sorted({*range(0, count, 97), count - 1}) if count > 2 else []
    small = count - len(big)

    def ints(*shape):
        return torch.randint(-8, 9, shape, generator=g, device="cuda").to(dt)

    As, Bs, Cs = ints(small, 8, 8), ints(small, 8, 8), torch.zeros((small, 8, 8), dtype=dt, device="cuda")
    Ab, Bb = ints(len(big), 72, 40), ints(len(big), 40, 136)
    Cb = torch.zeros((len(big), 72, 136), dtype=dt, device="cuda")
    probs, si, where = [], 0, set(big)
    a, b, c, A, B, C = (list(t.unbind(0)) for t in (As, Bs, Cs, Ab, Bb, Cb))
    for i in range(count):
        if i in where:
            at = i // 97 if i % 97 == 0 else len(big) - 1
            probs.append((A[at], B[at], C[at]))
        else:
            probs.append((a[si], b[si], c[si]))
            si += 1
    cc.grouped(probs, precision=precision)()
    assert torch.equal(Cs, As @ Bs) and torch.equal(Cb, Ab @ Bb)
    assert cc.device_status() == (cc.SUCCESS, 0)


@pytest.mark.parametrize("precision", ["bf16x3", "bf16x6"])
@pytest.mark.parametrize("copies", [1, 8, 60])
def test_prepass_depth(cuda, copies, precision):
    """Batches on both sides of the pre-pass's choice of row units and tiles a
    block (one copy takes some 65 blocks at the greater depth, 60 take 3900),
    with rows of more than one unit and column strips of one to many tiles."""
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(6)

    def ints(r, c):
        t = torch.zeros((r, -(-c // 4) * 4), device="cuda")
        t[:, :c] = torch.randint(-8, 9, (r, c), generator=g, device="cuda").float()
        return t[:, :c]

    shapes = [(300, 200, 701), (33, 70, 2113), (31, 65, 64), (100, 1, 257), (1, 129, 4099)]
    probs = [(ints(m, k), ints(k, n), ints(m, n)) for _ in range(copies) for m, n, k in shapes]
    cc.grouped(probs, precision=precision)()
    for A, B, C in probs:
        assert torch.equal(C, A @ B)  # integers: below 2^24, exact in any order
    assert cc.device_status() == (cc.SUCCESS, 0)
