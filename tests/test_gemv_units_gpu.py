"""The kernel of one to four rows where its plan has edges, and the norm that it takes itself."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def p(t, off=0):
    return C.c_void_p(t.data_ptr() + off)


def gemv(lib, kind, y, x, w, s, rows, n, k, g, s_off=0):
    if kind == 0:
        return lib.s2p_int8_gemv(p(y), p(x), p(w), p(s, s_off), rows, n, k, None)
    return (lib.s2p_intq_gemv if kind == 1 else lib.s2p_int4p_gemv)(p(y), p(x), p(w), p(s, s_off), rows, n, k, g, None)


def weights(kind, n, k, g, seed, pad=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randint(0, 256, (n, k // 2 if kind == 2 else k), dtype=torch.uint8, device="cuda", generator=gen)
    s = torch.rand(n * (1 if kind == 0 else k // g) + pad, device="cuda", generator=gen) * 0.01 + 0.001
    return w, s if kind == 0 else s.half(), gen


# n, k: several CTAs to an SM; sums that do not fit shared memory (the batch kernel's); either side of where three rows change kernels
@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("n,k", [(149, 512), (12345, 9728), (70001, 512), (5, 204800), (4733, 1024), (4737, 1024)])
def test_rows_equal_the_batch_kernels(mine, kind, n, k):
    w, s, gen = weights(kind, n, k, 32, n)
    x = torch.randn(5, k, device="cuda", generator=gen).bfloat16()
    want = torch.empty((5, n), dtype=torch.bfloat16, device="cuda")
    assert gemv(mine, kind, want, x, w, s, 5, n, k, 32) == 0
    for rows in (1, 2, 3, 4):
        got = torch.full((rows + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
        assert gemv(mine, kind, got, x, w, s, rows, n, k, 32) == 0
        torch.cuda.synchronize()
        assert torch.equal(got[:rows].view(torch.int16), want[:rows].view(torch.int16)) and (got[rows] == 7).all(), rows


# sums that fit shared memory, and two shapes whose do not (the batch kernel's, for one row too)
@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("f,k", [(77, 1024), (5, 409600), (70001, 1024)])
def test_swiglu_rows_equal_the_separate_kernels(testlib, kind, f, k):
    from _internal_abi import LinRef
    testlib.gemv_rows_swiglu.argtypes = [C.POINTER(LinRef), C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]
    w, s, gen = weights(kind, 2 * f, k, 32, f)
    x = torch.randn(5, k, device="cuda", generator=gen).bfloat16()
    gu, want = torch.empty((5, 2 * f), dtype=torch.bfloat16, device="cuda"), torch.empty((5, f), dtype=torch.bfloat16, device="cuda")
    assert gemv(testlib, kind, gu, x, w, s, 5, 2 * f, k, 32) == 0 and testlib.s2pk_silu_mul(p(gu), p(want), 5, f, None) == 0
    lin = LinRef(kind, w.data_ptr(), s.data_ptr(), 2 * f, k, 0 if kind == 0 else 5)
    for rows in (1, 2, 3, 4):
        got = torch.full((rows + 1, f), 7.0, dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        assert testlib.gemv_rows_swiglu(C.byref(lin), p(x), p(got), rows, None) == 0
        torch.cuda.synchronize()
        assert torch.equal(got[:rows].view(torch.int16), want[:rows].view(torch.int16)) and (got[rows] == 7).all(), rows


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("g,off", [(16, 0), (64, 2), (512, 0), (1024, 0), (2048, 6), (32, 2), (32, 14)])  # scales that 16-byte copies cannot take
def test_groups_and_unaligned_scales(mine, kind, g, off):
    n, k = 1031, 6144 if g > 512 else 1536  # groups shorter and longer than a tile
    w, s, gen = weights(kind, n, k, g, g + off, pad=8)
    x = torch.randn(5, k, device="cuda", generator=gen).bfloat16()
    want, got = (torch.empty((5, n), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert gemv(mine, kind, want, x, w, s, 5, n, k, g, off) == 0
    for rows in (1, 3):
        assert gemv(mine, kind, got, x, w, s, rows, n, k, g, off) == 0
        torch.cuda.synchronize()
        assert torch.equal(got[:rows].view(torch.int16), want[:rows].view(torch.int16)), rows


@pytest.mark.parametrize("kind", ["int8", "int8_grouped", "int4"])
def test_every_kind_of_activation_gives_the_oracles_bits(mine, oracle, kind):
    """Subnormals, signed zeros, infinities and NaN: the mixed fma takes bf16 as fmaf takes its f32."""
    from oracle import oracle_api
    n, k = 67, 1024
    rng = np.random.default_rng(3)
    w = rng.integers(0, 256, size=(n, k // 2 if kind == "int4" else k), dtype=np.uint8)
    s = rng.random((n, 1 if kind == "int8" else k // 32), dtype=np.float32) * 0.01 + 0.001
    s = s if kind == "int8" else s.astype(np.float16)
    x = oracle_api.f32_to_bf16(rng.standard_normal((16, k), dtype=np.float32))
    x[0] = rng.integers(0, 0x80, k) | (rng.integers(0, 2, k) << 15)          # subnormals and zeros alone
    x[1] = (x[1] & 0x807F) | (rng.integers(0, 40, k) << 7)                   # small enough for subnormal products and sums
    x[2, ::7] = x[2, ::7] & 0x807F                                           # subnormals among ordinary values
    x[3, 5] = 0x7F80                                                         # an infinity
    x[4, 9], x[4, 700] = 0xFF80, 0x7F80                                      # two that cancel
    x[5, 33] = 0x7FC1                                                        # a NaN
    x[6] = 0x8000                                                            # minus zero alone
    x[7] = (x[7] & 0x807F) | (rng.integers(0xF0, 0xFF, k) << 7)              # overflowing sums
    want = np.empty((16, n), np.uint16)
    args = [oracle_api.ptr(a) for a in (want, x, w, s)] + [16, n, k]
    oracle.s2po_gemv_int8(*args) if kind == "int8" else (oracle.s2po_gemv_g if kind == "int8_grouped" else oracle.s2po_gemv_p)(*args, 32)
    dw, ds, dx = (torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a).cuda() for a in (w, s, x))
    code = {"int8": 0, "int8_grouped": 1, "int4": 2}[kind]
    is_nan = lambda v: (v & 0x7FFF) > 0x7F80  # noqa: E731
    for rows in (1, 2, 4, 5, 8, 16):
        for first in range(0, 16 - rows + 1, rows):
            y = torch.empty((rows, n), dtype=torch.bfloat16, device="cuda")
            assert gemv(mine, code, y, dx[first:].contiguous(), dw, ds, rows, n, k, 32) == 0
            got, ref = y.view(torch.int16).cpu().numpy().view(np.uint16), want[first:first + rows]
            assert ((got == ref) | (is_nan(got) & is_nan(ref))).all(), (rows, first)


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("rows", [1, 2])
@pytest.mark.parametrize("n,swiglu", [(6144, 0), (150, 0), (2 * 9728, 1), (2 * 77, 1)])
def test_norm_in_the_linear_equals_the_two_kernels(testlib, kind, rows, n, swiglu):
    from _internal_abi import LinRef, NormIn
    P, I, L = C.c_void_p, C.c_int, C.POINTER(LinRef)
    testlib.gemv_rows.argtypes, testlib.gemv_rows_swiglu.argtypes = [L, P, P, I, I, P], [L, P, P, I, P]
    testlib.gemv_rows_norm.argtypes = [L, C.POINTER(NormIn), P, I, I, P]
    testlib.add_norm_to.argtypes = [P, P, P, P, P, I, P]
    k = 2560
    w, s, gen = weights(kind, n, k, 32, n + rows)
    lin = LinRef(kind, w.data_ptr(), s.data_ptr(), n, k, 0 if kind == 0 else 5)
    src, add = (torch.randn(rows, k, device="cuda", generator=gen).bfloat16() for _ in range(2))
    gain = (torch.rand(k, device="cuda", generator=gen) + 0.5).bfloat16()
    outs = n // 2 if swiglu else n
    x, x_want, norm = (torch.empty_like(src) for _ in range(3))
    want, got = (torch.empty((rows, outs), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    assert testlib.add_norm_to(p(src), p(add), p(x_want), p(gain), p(norm), rows, None) == 0
    assert (testlib.gemv_rows_swiglu(C.byref(lin), p(norm), p(want), rows, None) if swiglu else testlib.gemv_rows(C.byref(lin), p(norm), p(want), rows, 0, None)) == 0
    nm = NormIn(src.data_ptr(), add.data_ptr(), gain.data_ptr(), x.data_ptr(), 1e-6, 0)
    assert testlib.gemv_rows_norm(C.byref(lin), C.byref(nm), p(got), swiglu, rows, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(x.view(torch.int16), x_want.view(torch.int16)) and torch.equal(got.view(torch.int16), want.view(torch.int16))
    nm.x_out = src.data_ptr()  # every CTA reads src: it cannot be written
    assert testlib.gemv_rows_norm(C.byref(lin), C.byref(nm), p(got), swiglu, rows, None) != 0


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_weights_written_by_the_kernel_in_front(mine, kind):
    """A linear starts while the kernel in front of it finishes: weights that this one writes are waited for all the same."""
    n, k, gen = 4864, 1024, torch.Generator(device="cuda").manual_seed(kind)
    per_row = k // 4 if kind == 2 else k // 2  # bf16 values whose bytes are a row of weights
    gu = torch.randn((n, 2 * per_row), device="cuda", generator=gen).bfloat16()
    x = torch.randn((9, k), device="cuda", generator=gen).bfloat16()
    _, s, _ = weights(kind, n, k, 32, 5)
    w, got, want = torch.empty((n, per_row), dtype=torch.bfloat16, device="cuda"), *(torch.empty((9, n), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert mine.s2pk_silu_mul(p(gu), p(w), n, per_row, None) == 0
    torch.cuda.synchronize()
    for rows in (1, 2, 3, 8, 9):
        assert gemv(mine, kind, want, x, w, s, rows, n, k, 32) == 0
        for _ in range(20):
            w.view(torch.int16).fill_(0x1111)
            torch.cuda.synchronize()
            assert mine.s2pk_silu_mul(p(gu), p(w), n, per_row, None) == 0 and gemv(mine, kind, got, x, w, s, rows, n, k, 32) == 0
            torch.cuda.synchronize()
            assert torch.equal(got[:rows].view(torch.int16), want[:rows].view(torch.int16)), rows


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_activations_written_by_the_kernel_in_front(mine, kind):
    """The same for the activations, which every caller's chain writes just before: SwiGLU, linear, SwiGLU, each reading the one in front."""
    n, k, gen = 4864, 9728, torch.Generator(device="cuda").manual_seed(7 + kind)
    w, s, _ = weights(kind, n, k, 32, 9)
    gu = torch.randn((9, 2 * k), device="cuda", generator=gen).bfloat16()
    bufs = [torch.empty((9, c), dtype=torch.bfloat16, device="cuda") for c in (k, n, n // 2)]  # x, y, h
    for rows in (1, 2, 3, 8, 9):
        def chain(wait):
            x, y, h = bufs
            assert mine.s2pk_silu_mul(p(gu), p(x), rows, k, None) == 0
            wait()
            assert gemv(mine, kind, y, x, w, s, rows, n, k, 32) == 0
            wait()
            assert mine.s2pk_silu_mul(p(y), p(h), rows, n // 2, None) == 0
            torch.cuda.synchronize()
        chain(torch.cuda.synchronize)
        want = [b[:rows].clone() for b in bufs]
        for _ in range(20):
            for b in bufs:
                b.view(torch.int16).fill_(0x4111)
            torch.cuda.synchronize()
            chain(lambda: None)
            assert all(torch.equal(b[:rows].view(torch.int16), v.view(torch.int16)) for b, v in zip(bufs, want)), rows
