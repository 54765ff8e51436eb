"""One row through the linear against a plain fp32 product, and against itself as the first of two rows: the same bits."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("n,k", [(1, 512), (3, 2560), (1029, 4608), (2561, 9728), (6146, 1536), (19457, 1024)])  # shared, two tiles, one tile at a time
def test_one_row(mine, kind, n, k):
    g = torch.Generator(device="cuda").manual_seed(n)
    codes = torch.randint(-8 if kind == 2 else -127, 8 if kind == 2 else 128, (n, k), device="cuda", generator=g)
    w = ((codes[:, 0::2] & 15) | ((codes[:, 1::2] & 15) << 4)).to(torch.uint8) if kind == 2 else codes.to(torch.int8)
    s = torch.rand(n, 1 if kind == 0 else k // 32, device="cuda", generator=g) * 0.01 + 0.001
    s = s if kind == 0 else s.half()
    x = torch.randn(2, k, device="cuda", generator=g).bfloat16()
    one, two = torch.full((n + 1,), 7.0, dtype=torch.bfloat16, device="cuda"), torch.empty((2, n), dtype=torch.bfloat16, device="cuda")
    for y, m in ((one, 1), (two, 2)):
        args = (p(y), p(x), p(w), p(s), m, n, k)
        assert (mine.s2p_int8_gemv(*args, None) if kind == 0 else (mine.s2p_intq_gemv if kind == 1 else mine.s2p_int4p_gemv)(*args, 32, None)) == 0
    torch.cuda.synchronize()
    assert torch.equal(one[:n].view(torch.int16), two[0].view(torch.int16)) and one[n] == 7
    full = codes.double() * (s.double() if kind == 0 else s.double().repeat_interleave(32, 1))
    want = full @ x[0].double()
    assert ((one[:n].double() - want).abs() <= 0.01 * want.abs() + 1e-3 * want.abs().max()).all()


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("rows", [1, 2, 3, 4])
@pytest.mark.parametrize("ffn,k", [(1, 512), (515, 2560), (9728, 1536)])
def test_swiglu_in_the_linear_equals_the_two_kernels(testlib, kind, rows, ffn, k):
    from _internal_abi import LinRef
    P, I, L = C.c_void_p, C.c_int, C.POINTER(LinRef)
    testlib.gemv_rows.argtypes, testlib.gemv_rows_swiglu.argtypes = [L, P, P, I, I, P], [L, P, P, I, P]
    testlib.silu_mul.argtypes = [P, P, I, I, P]
    g = torch.Generator(device="cuda").manual_seed(ffn + rows)
    w = torch.randint(0, 256, (2 * ffn, k // 2 if kind == 2 else k), dtype=torch.uint8, device="cuda", generator=g)
    s = torch.rand(2 * ffn, 1 if kind == 0 else k // 32, device="cuda", generator=g) * 0.002 + 0.001
    s = s if kind == 0 else s.half()
    x = torch.randn(rows, k, device="cuda", generator=g).bfloat16()
    lin = LinRef(kind, w.data_ptr(), s.data_ptr(), 2 * ffn, k, 0 if kind == 0 else 5)
    gu = torch.empty((rows, 2 * ffn), dtype=torch.bfloat16, device="cuda")
    want, got = torch.empty((rows, ffn), dtype=torch.bfloat16, device="cuda"), torch.full((rows + 1, ffn), 7.0, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    assert testlib.gemv_rows(C.byref(lin), p(x), p(gu), rows, 0, None) == 0 and testlib.silu_mul(p(gu), p(want), rows, ffn, None) == 0
    assert testlib.gemv_rows_swiglu(C.byref(lin), p(x), p(got), rows, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(got[:rows].view(torch.int16), want.view(torch.int16)) and (got[rows] == 7).all()
