"""The thin kernel's rounding errors: no larger than those of the form with
four CTAs an SM and four (FP64: two) consecutive k a lane, whose rms errors on
the same kind of operands, relative to the rms of the result, are given here
(errors pooled over seeds, a thousand or more, known to 3 %)."""
import pytest

import cucosma_b200 as cc

pytestmark = pytest.mark.gpu

# (m, n, k), dtype, rms relative error of that form, seeds
CASES = [((5, 30000, 100), "float32", 7.17e-8, 1), ((5, 30000, 100), "float64", 1.01e-16, 1),
         ((20000, 7, 200), "float32", 7.65e-8, 1), ((20000, 7, 200), "float64", 1.19e-16, 1),
         ((4, 8, 3000), "float32", 1.05e-7, 200), ((4, 8, 3000), "float64", 1.70e-16, 200),
         ((1, 4096, 4096), "float32", 1.03e-7, 3), ((1, 4096, 4096), "float64", 1.65e-16, 3),
         ((64, 5, 5000), "float32", 1.16e-7, 40), ((8, 8, 40000), "float32", 1.10e-7, 150),
         ((12, 7, 1435677), "float64", 2.47e-16, 20), ((8, 16, 3000000), "float32", 1.67e-7, 20),
         ((8, 16, 3000000), "float64", 2.79e-16, 20), ((1, 16, 1570806), "float32", 1.39e-7, 40)]


@pytest.mark.parametrize("shape,dtype,limit,seeds", CASES, ids=["%dx%dx%d-%s" % (c[0] + (c[1],)) for c in CASES])
def test_thin_rounding(cuda, shape, dtype, limit, seeds):
    import torch

    m, n, k = shape
    dt = getattr(torch, dtype)
    err2 = ref2 = 0.0
    for seed in range(seeds):
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)

        def ints(r, c, top):
            v = 16 // dt.itemsize
            t = torch.zeros((r, -(-c // v) * v), dtype=dt, device="cuda")
            t[:, :c] = torch.randint(-top, top, (r, c), generator=g, device="cuda").to(dt)
            return t[:, :c]

        # integers: exact results by 64-bit products of at most 2^53
        top = 2**24 if dt is torch.float32 else 2**26
        A, B, C = ints(m, k, top), ints(k, n, top), ints(m, n, 1)
        cc.cosma_sgemm(A, B, C, 1.0, 0.0)
        Ad, Bd = A.double(), B.double()
        hi = torch.round(Ad / 8192)
        lo = Ad - 8192 * hi
        ph = torch.zeros((m, n), dtype=torch.int64, device="cuda")
        pl = torch.zeros_like(ph)
        for k0 in range(0, k, 8192):  # |hi * b|, |lo * b| < 2^39
            ph += (hi[:, k0:k0 + 8192] @ Bd[k0:k0 + 8192]).to(torch.int64)
            pl += (lo[:, k0:k0 + 8192] @ Bd[k0:k0 + 8192]).to(torch.int64)
        ref = ph.double() * 8192
        err2 += float(((C.double() - ref) - pl.double()).pow(2).sum())
        ref2 += float(ref.pow(2).sum())
    samples = seeds * m * n
    # the limit's own sampling error and this sample's, three deviations of each
    assert (err2 / ref2) ** 0.5 <= limit * (1 + 0.03 + 3 / (2 * samples) ** 0.5)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("k", [100, 70001])
def test_infinities_and_nan(cuda, dtype, k):
    """Infinite and NaN products reach their outputs, and no others, through every step of the reduction."""
    import torch

    dt = getattr(torch, dtype)
    m, n = 6, 8
    A = torch.zeros((m, -(-k // 4) * 4), dtype=dt, device="cuda")[:, :k]
    B = torch.ones((k, n), dtype=dt, device="cuda")
    A.fill_(0.5)
    inf = float("inf")
    A[1, 0], A[2, k - 1], A[3, 17], A[4, 33], A[4, k - 2] = inf, -inf, float("nan"), inf, -inf
    A[5, 64] = torch.finfo(dt).max
    C = torch.zeros((m, n), dtype=dt, device="cuda")
    cc.cosma_sgemm(A, B, C, 1.0, 0.0)
    want = torch.tensor([0.5 * k, inf, -inf, float("nan"), float("nan"), torch.finfo(dt).max], dtype=dt, device="cuda")
    assert torch.equal(C.isnan(), want.isnan()[:, None].expand(m, n))
    ok = [0, 1, 2, 5]
    assert torch.equal(C[ok], want[ok, None].expand(len(ok), n))
