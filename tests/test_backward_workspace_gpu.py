"""Workspace the backward pass asks for: both products' planes, the larger one's
where both would take much of the memory."""
import ctypes as C

import pytest

import cucosma_b200 as cc

pytestmark = pytest.mark.gpu


def query(m, n, k, precision="bf16x3", epilogue="sigmoid"):
    d = cc.GemmDesc()
    cc.lib().cucosma_gemm_desc_init(C.byref(d))
    d.m, d.n, d.k = m, n, k
    d.lda, d.ldb, d.ldc = (-(-x // 4) * 4 for x in (k, n, n))
    d.precision, d.epilogue = cc.PRECISIONS[precision], cc.EPILOGUES[epilogue]
    size = C.c_size_t(0)
    assert cc.lib().cucosma_gemm_backward_workspace_size(C.byref(d), C.byref(size)) == cc.SUCCESS
    return size.value


@pytest.mark.parametrize("precision,terms", [("bf16x3", 2), ("bf16x6", 3)])
def test_query(cuda, precision, terms):
    # planes of one product of N^3: G and the other operand, 2 * terms bytes a value
    n = 4096
    assert query(n, n, n, precision) >= 2 * (2 * n * n * 2 * terms)
    n = 60000  # six matrices of 14.4 GB; with both products' planes (58 or 86 GB) they would not fit
    assert query(n, n, n, precision) < 1.05 * (2 * n * n * 2 * terms)
