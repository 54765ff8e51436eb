"""The batched linear from resident f16 tiles against the one that converts as it goes: the same bits."""
import ctypes as C

import pytest

from _internal_abi import LinRef

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class WidePart(C.Structure):
    _fields_ = [("partial", C.c_void_p), ("scales", C.c_void_p), ("pieces", C.c_int), ("M", C.c_int)]


@pytest.fixture(scope="module")
def tl(testlib):
    P, I = C.c_void_p, C.c_int
    L = C.POINTER(LinRef)
    for name, args in (("skinny_setup", [I]), ("skinny_gemm_tc", [L, P, I, P, P, P]), ("skinny_gemm_tc_swiglu", [L, P, I, P, P]),
                       ("wide_weight_bytes", [L, I]), ("wide_convert", [L, I, P, P]), ("wide_pack", [I, P, I, I, P, P]),
                       ("wide_gemm", [L, P, P, I, I, P, P, I, C.POINTER(WidePart), P]),
                       ("wide_norm", [P, C.POINTER(WidePart), P, P, P, P, P, I, I, P])):
        getattr(testlib, name).argtypes = args
    testlib.wide_weight_bytes.restype = C.c_size_t
    assert testlib.skinny_setup(256) == 0
    return testlib


def p(t):
    return C.c_void_p(t.data_ptr())


def linear(kind, n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randint(0, 256, (n, k // 2 if kind == 2 else k), dtype=torch.uint8, device="cuda", generator=g)
    s = torch.rand(n, 1 if kind == 0 else k // 32, device="cuda", generator=g) * 0.01 + 0.001
    s = s if kind == 0 else s.half()
    return LinRef(kind, w.data_ptr(), s.data_ptr(), n, k, 0 if kind == 0 else 5), (w, s)


def tiles(tl, lin, ffn):
    out = torch.empty(tl.wide_weight_bytes(C.byref(lin), ffn), dtype=torch.uint8, device="cuda")
    assert tl.wide_convert(C.byref(lin), ffn, p(out), None) == 0
    return out


def units(tl, kind, x):
    xt = torch.full((256 * x.shape[1],), float("nan"), dtype=torch.float16, device="cuda")  # padding must not leak
    assert tl.wide_pack(kind, p(x), x.shape[0], x.shape[1], p(xt), None) == 0
    return xt


@pytest.mark.parametrize("kind", [2, 0, 1])
@pytest.mark.parametrize("rows,n,k", [(17, 2560, 4096), (1, 2560, 512), (128, 2560, 1024), (129, 2560, 2560), (256, 2560, 768)])
def test_split_outputs_through_the_norm_that_adds_them(tl, mine, kind, rows, n, k):
    lin, keep = linear(kind, n, k, rows)
    g = torch.Generator(device="cuda").manual_seed(k)
    x, r, gain = (torch.randn(*s, device="cuda", generator=g).bfloat16() for s in ((rows, k), (rows, n), (n,)))
    want = r.clone()
    assert tl.skinny_gemm_tc(C.byref(lin), p(x), rows, p(want), p(want), None) == 0
    y_want = torch.empty_like(r)
    assert mine.s2pk_rms_norm(p(want), p(gain), p(y_want), rows, n, 1e-6, None) == 0
    part, alt = WidePart(), torch.empty_like(r)
    assert tl.wide_gemm(C.byref(lin), p(tiles(tl, lin, 0)), p(units(tl, kind, x)), rows, 0, p(alt), None, 0, C.byref(part), None) == 0
    y, t = torch.empty_like(r), torch.full((256 * n,), float("nan"), dtype=torch.float16, device="cuda")
    assert tl.wide_norm(p(r), C.byref(part), p(alt), p(r), p(gain), p(y), p(t), kind, rows, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(r.view(torch.int16), want.view(torch.int16))
    assert torch.equal(y.view(torch.int16), y_want.view(torch.int16))
    packed = units(tl, kind, y)  # the units the norm left are those of its bf16 result
    nb = max(16, 1 << (rows - 1).bit_length())
    a, b = (v[:nb * n].view(n // 8, nb, 8)[:, :rows] for v in (t, packed))
    assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("kind", [2, 0])
@pytest.mark.parametrize("rows", [17, 130])
def test_outputs_of_a_matrix_that_is_not_split(tl, kind, rows):
    n, k = 100 * 128 - 3, 256
    lin, keep = linear(kind, n, k, 3)
    x = torch.randn(rows, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4)).bfloat16()
    want, got = (torch.zeros(rows, n, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert tl.skinny_gemm_tc(C.byref(lin), p(x), rows, p(want), None, None) == 0
    part = WidePart()
    assert tl.wide_gemm(C.byref(lin), p(tiles(tl, lin, 0)), p(units(tl, kind, x)), rows, 0, p(got), None, 0, C.byref(part), None) == 0
    torch.cuda.synchronize()
    assert not part.partial and torch.equal(got.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("kind", [2, 0, 1])
@pytest.mark.parametrize("rows,ffn,k", [(17, 200, 512), (32, 9728, 512), (100, 4808, 256), (129, 9664, 1024), (256, 9728, 256)])
def test_swiglu_as_rows_and_as_units(tl, kind, rows, ffn, k):
    """No tile split, all of them, and the surplus beyond one per SM (split 10, 4 or not at all by K)."""
    lin, keep = linear(kind, 2 * ffn, k, ffn)
    x = torch.randn(rows, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)).bfloat16()
    want, got = (torch.zeros(rows, ffn, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert tl.skinny_gemm_tc_swiglu(C.byref(lin), p(x), rows, p(want), None) == 0
    w, xt = tiles(tl, lin, ffn), units(tl, kind, x)
    assert tl.wide_gemm(C.byref(lin), p(w), p(xt), rows, ffn, p(got), None, 0, None, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    if ffn % 64 == 0:
        t = torch.full((256 * ffn,), float("nan"), dtype=torch.float16, device="cuda")
        assert tl.wide_gemm(C.byref(lin), p(w), p(xt), rows, ffn, None, p(t), kind, None, None) == 0
        nb = max(16, 1 << (rows - 1).bit_length())
        a, b = (v[:nb * ffn].view(ffn // 8, nb, 8)[:, :rows] for v in (t, units(tl, kind, want)))
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
