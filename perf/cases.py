"""Performance cases of the library: the GEMM calls its users make, through the
public Python entry points (which pass straight to the C ABI), with operands
resident on the GPU.

Three kinds of case:

  gemm     one call, C <- epi(alpha*A@B + beta*C).  entry "cosma" is the
           reference-shaped call (native arithmetic, library-managed
           workspace); entry "gemm" is the descriptor call with a precision
           form, an epilogue and a workspace the caller keeps.
  grouped  one launch of a plan over `count` independent GEMMs of uneven sizes
           (M, N log-uniform in [64, 2048], K log-uniform in [64, 8192], the
           batch drawn from `shape_seed`).
  train    forward Y = epi(A@B) and the backward pass to dA and dB.

Every matrix is row-major with rows padded to 16 bytes, as the API asks.
"""
import math
import random

import torch

import cucosma_b200 as cc

F32, F64 = "float32", "float64"


def _gemm(name, m, n, k, dtype=F32, precision="native", entry="gemm", beta=0.0, epilogue="none", values="uniform"):
    return {"name": name, "kind": "gemm", "m": m, "n": n, "k": k, "dtype": dtype, "precision": precision,
            "entry": entry, "alpha": 1.0, "beta": beta, "epilogue": epilogue, "values": values}


def listed():
    return [
        # The drop-in call on a small block: launch latency and host work.
        _gemm("sgemm_small", 200, 136, 96, entry="cosma"),
        # Plain SGEMM at 1024^3, the reference's own verification size.
        _gemm("sgemm_1024", 1024, 1024, 1024, entry="cosma"),
        # The reference's special list: a tiny C, a very long K.
        _gemm("sgemm_thin_long_k", 4, 8, 3000000, entry="cosma"),
        # The FP64 drop-in on odd sizes, accumulating into C.
        _gemm("dgemm_ragged", 1000, 777, 1531, dtype=F64, entry="cosma", beta=0.5),
        # The FP32-accurate tensor-core form at its headline size.
        _gemm("bf16x6_8192", 8192, 8192, 8192, precision="bf16x6"),
        # The same form at an ordinary size with odd edges and an activation
        # (a layer of a network whose widths are no multiple of a tile).
        _gemm("bf16x6_ragged_sigmoid", 1234, 1111, 777, precision="bf16x6", epilogue="sigmoid"),
        # Flat family: a short K updates a large C (rank-K update).
        _gemm("bf16x3_flat", 16384, 16384, 256, precision="bf16x3", beta=0.5),
        # Large-K family: a small C from a million-long contraction.
        _gemm("bf16x6_large_k", 256, 256, 1048576, precision="bf16x6", beta=0.5),
        # Large-N family with the fused sigmoid: a wide batch through a layer.
        _gemm("bf16x3_large_n_sigmoid", 256, 1048576, 256, precision="bf16x3", beta=0.5, epilogue="sigmoid"),
        # DGEMM by INT8 slices, slice count chosen on the device (the default).
        _gemm("ozaki_4096", 4096, 4096, 4096, dtype=F64, precision="ozaki"),
        # Uneven batch in one launch: 512 GEMMs.
        {"name": "grouped_bf16x3_512", "kind": "grouped", "count": 512, "shape_seed": 5, "precision": "bf16x3",
         "dtype": F32},
        # Forward and backward of a sigmoid layer.
        {"name": "train_4096_sigmoid", "kind": "train", "m": 4096, "n": 4096, "k": 4096, "precision": "bf16x3",
         "epilogue": "sigmoid"},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _size(rng, lo, hi):
    """Log-uniform; half of the sizes as drawn (mostly odd ones), half rounded to a multiple of 32."""
    v = _log(rng, lo, hi)
    return v if rng.random() < 0.5 or v < 64 else v // 32 * 32


def draw(rng):
    what = rng.choice(["small", "native", "thin", "double", "tensor", "tensor", "flat", "large_k", "large_n", "ozaki",
                       "grouped", "train"])
    beta = rng.choice([0.0, 0.5])
    epilogue = rng.choice(["none", "none", "sigmoid", "relu"])
    bf16 = rng.choice(["bf16x3", "bf16x6"])
    if what == "small":
        c = _gemm("", _size(rng, 17, 400), _size(rng, 17, 400), _size(rng, 17, 400), entry="cosma", beta=beta)
    elif what == "native":
        c = _gemm("", _size(rng, 256, 3000), _size(rng, 256, 3000), _size(rng, 256, 3000), entry="cosma", beta=beta)
    elif what == "thin":
        # a thin side against a long K or a long N
        thin, other, long_ = rng.randint(1, 8), rng.randint(1, 16), _log(rng, 30000, 3000000)
        m, n, k = rng.choice([(thin, other, long_), (other, thin, long_), (thin, long_, other)])
        c = _gemm("", m, n, k, dtype=rng.choice([F32, F32, F64]), entry="cosma", beta=beta)
    elif what == "double":
        c = _gemm("", _size(rng, 100, 2000), _size(rng, 100, 2000), _size(rng, 100, 2000), dtype=F64, entry="cosma",
                  beta=beta)
    elif what == "tensor":
        # ordinary layers up to the headline size
        c = _gemm("", _size(rng, 128, 8192), _size(rng, 128, 8192), _size(rng, 128, 8192), precision=bf16, beta=beta,
                  epilogue=epilogue)
    elif what == "flat":
        c = _gemm("", _size(rng, 4096, 16384), _size(rng, 4096, 16384), _size(rng, 64, 256), precision=bf16,
                  beta=beta, epilogue=epilogue)
    elif what == "large_k":
        c = _gemm("", _size(rng, 130, 256), _size(rng, 130, 256), _size(rng, 16384, 1048576), precision=bf16,
                  beta=beta)
    elif what == "large_n":
        c = _gemm("", _size(rng, 130, 256), _size(rng, 16384, 1048576), _size(rng, 130, 256), precision=bf16,
                  beta=beta, epilogue=epilogue)
    elif what == "ozaki":
        # now and then entries whose exponents are spread widely
        c = _gemm("", _size(rng, 256, 4096), _size(rng, 256, 4096), _size(rng, 256, 4096), dtype=F64,
                  precision="ozaki", beta=beta, values="spread" if rng.random() < 0.2 else "uniform")
    elif what == "grouped":
        p = rng.choice(["bf16x3", "bf16x6", "ozaki"])
        c = {"kind": "grouped", "count": _log(rng, 16, 512 if p == "bf16x3" else 256),
             "shape_seed": rng.randrange(1 << 20), "precision": p, "dtype": F64 if p == "ozaki" else F32}
    else:
        c = {"kind": "train", "m": _size(rng, 512, 4096), "n": _size(rng, 512, 4096), "k": _size(rng, 512, 4096),
             "precision": bf16, "epilogue": rng.choice(["sigmoid", "relu", "none"])}
    c.pop("name", None)
    return c


def _shapes(case):
    rng = random.Random(case["shape_seed"])
    return [(_log(rng, 64, 2048), _log(rng, 64, 2048), _log(rng, 64, 8192)) for _ in range(case["count"])]


def _pitch(cols, dtype):
    vec = 16 // dtype.itemsize
    return -(-cols // vec) * vec


def _matrix(rows, cols, dtype, gen, scale=1.0, values="uniform"):
    """rows x cols view of a row-major buffer with 16-byte rows, entries uniform in
    [-scale, scale], or sign * exp(N(0, 8^2))."""
    t = torch.empty((rows, _pitch(cols, dtype)), dtype=dtype, device="cuda")
    if values == "spread":
        t.normal_(0.0, 8.0, generator=gen).exp_()
        t *= torch.randint(0, 2, t.shape, device="cuda", generator=gen) * 2 - 1
    else:
        t.uniform_(-scale, scale, generator=gen)
    return t[:, :cols]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _operands(case, seed):
    g, dt = _gen(seed), getattr(torch, case["dtype"])
    A = _matrix(case["m"], case["k"], dt, g, values=case["values"])
    B = _matrix(case["k"], case["n"], dt, g, values=case["values"])
    C = _matrix(case["m"], case["n"], dt, g)
    return A, B, C


def _batch(case, seed):
    """The batch's operands, and one flat buffer that holds every C (zeroed, so that row padding is defined)."""
    g, dt = _gen(seed), getattr(torch, case["dtype"])
    shapes = _shapes(case)
    elems = sum(m * _pitch(k, dt) + k * _pitch(n, dt) for m, n, k in shapes)
    src = torch.empty(elems, dtype=dt, device="cuda").uniform_(-1.0, 1.0, generator=g)
    flat = torch.zeros(sum(m * _pitch(n, dt) for m, n, k in shapes), dtype=dt, device="cuda")
    at, ct, problems = 0, 0, []

    def take(buf, at, rows, cols):
        ld = _pitch(cols, dt)
        return buf[at:at + rows * ld].view(rows, ld)[:, :cols], at + rows * ld

    for m, n, k in shapes:
        A, at = take(src, at, m, k)
        B, at = take(src, at, k, n)
        C, ct = take(flat, ct, m, n)
        problems.append((A, B, C))
    return problems, flat


def _train_operands(case, seed):
    g = _gen(seed)
    A = _matrix(case["m"], case["k"], torch.float32, g, 0.1)
    B = _matrix(case["k"], case["n"], torch.float32, g, 0.1)
    dY = _matrix(case["m"], case["n"], torch.float32, g)
    return A, B, dY


def prepare(case, seed):
    if case["kind"] == "gemm":
        A, B, C = _operands(case, seed)
        s = {"case": case, "A": A, "B": B, "C": C}
        if case["entry"] == "gemm":
            d = cc.make_desc(A, B, C, case["alpha"], case["beta"], precision=case["precision"],
                             epilogue=case["epilogue"])
            s["ws"] = cc.alloc_workspace(d)
        return s
    if case["kind"] == "grouped":
        problems, flat = _batch(case, seed)
        return {"case": case, "plan": cc.grouped(problems, precision=case["precision"]), "flat": flat}
    A, B, dY = _train_operands(case, seed)
    m, n, k = case["m"], case["n"], case["k"]
    Y = torch.empty((m, _pitch(n, A.dtype)), device="cuda")[:, :n]
    dA = torch.empty((m, _pitch(k, A.dtype)), device="cuda")[:, :k]
    dB = torch.empty((k, _pitch(n, A.dtype)), device="cuda")[:, :n]
    ws = cc.alloc_workspace(cc.make_desc(A, B, Y, precision=case["precision"], epilogue=case["epilogue"]))
    return {"case": case, "A": A, "B": B, "dY": dY, "Y": Y, "dA": dA, "dB": dB, "ws": ws}


def run(s):
    c = s["case"]
    if c["kind"] == "grouped":
        s["plan"]()
        return s["flat"]
    if c["kind"] == "train":
        cc.gemm(s["A"], s["B"], s["Y"], precision=c["precision"], epilogue=c["epilogue"], workspace=s["ws"])
        cc.gemm_backward(s["A"], s["B"], s["Y"], s["dY"], s["dA"], s["dB"], precision=c["precision"],
                         epilogue=c["epilogue"])
        return {"Y": s["Y"], "dA": s["dA"], "dB": s["dB"]}
    if c["entry"] == "cosma":
        return cc.cosma_sgemm(s["A"], s["B"], s["C"], c["alpha"], c["beta"])
    return cc.gemm(s["A"], s["B"], s["C"], c["alpha"], c["beta"], precision=c["precision"], epilogue=c["epilogue"],
                   workspace=s["ws"])


def work(case):
    """Each operand read once, each output written once (C also read when beta is not 0); 2*M*N*K flops a product."""
    if case["kind"] == "grouped":
        es = 8 if case["dtype"] == F64 else 4
        shapes = _shapes(case)
        return {"bytes": es * sum(m * k + k * n + m * n for m, n, k in shapes),
                "flops": 2 * sum(m * n * k for m, n, k in shapes)}
    m, n, k = case["m"], case["n"], case["k"]
    if case["kind"] == "train":
        return {"bytes": 4 * (2 * m * k + 2 * k * n + 2 * m * n), "flops": 6 * m * n * k}
    es = 8 if case["dtype"] == F64 else 4
    return {"bytes": es * (m * k + k * n + m * n * (2 if case["beta"] else 1)), "flops": 2 * m * n * k}


def _epi(z, epilogue):
    return torch.sigmoid(z) if epilogue == "sigmoid" else z.clamp_min(0) if epilogue == "relu" else z


def exact(case, seed):
    """The same results from torch in 64 bits."""
    if case["kind"] == "grouped":
        problems, flat = _batch(case, seed)
        out, at = torch.zeros(flat.numel(), dtype=torch.float64, device="cuda"), 0
        for A, B, C in problems:
            rows, ld = C.shape[0], C.stride(0) if C.shape[0] > 1 else _pitch(C.shape[1], C.dtype)
            out[at:at + rows * ld].view(rows, ld)[:, :C.shape[1]] = A.double() @ B.double()
            at += rows * ld
        return out
    if case["kind"] == "train":
        A, B, dY = (t.double() for t in _train_operands(case, seed))
        Y = _epi(A @ B, case["epilogue"])
        G = dY * (Y * (1 - Y) if case["epilogue"] == "sigmoid" else (Y > 0) if case["epilogue"] == "relu" else 1.0)
        return {"Y": Y, "dA": G @ B.T, "dB": A.T @ G}
    A, B, C = _operands(case, seed)
    z = A.double() @ B.double()
    z *= case["alpha"]
    if case["beta"]:
        z += case["beta"] * C.double()
    return _epi(z, case["epilogue"])
