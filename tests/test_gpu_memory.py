"""With little memory left a large product's operand planes, which the context keeps for the
next one, must not make a later call fail that fits without them."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dp(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def test_planes_give_way():
    import tngpu as tn
    torch = pytest.importorskip("torch")
    ctx = tn.context()
    n = 4096
    A, out, one = np.ones((n, n), complex, order="F"), np.zeros((n, n), complex, order="F"), np.ones(1, complex)
    big = 16384
    B, x, y = np.zeros((big, big), complex, order="F"), np.ones(big, complex), np.zeros(big, complex)
    B[:, 0] = 2.0
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - (6 << 30), dtype=torch.uint8, device="cuda")
    try:
        # 2.7 GB of planes beside 1.3 GB of operands, then 4.3 GB of operand
        ctx.check(ctx.lib.tn_gate2_apply(ctx.h, n, n, n, 1, dp(A), dp(A), dp(one), dp(out)))
        assert np.all(out == n)
        ctx.check(ctx.lib.tn_gemm(ctx.h, big, 1, big, dp(B), 0, dp(x), dp(y), 0))
        assert np.all(y == 2.0)
    finally:
        del hog
        torch.cuda.empty_cache()
