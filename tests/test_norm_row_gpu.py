"""The norm fused with what precedes it (residual add, embedding lookup, arg-max) against the separate launchers."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
D, CB, EPS = 2560, 4096, 1e-6


@pytest.fixture
def tools(mine, testlib):
    import torch
    for name, n in (("add_norm", 6), ("copy_norm", 6), ("embed_norm", 9)):
        getattr(testlib, name).argtypes = [C.c_void_p] * (n - 2) + [C.c_int, C.c_void_p]
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731

    def scalar_norm(x, w):
        """The element-wise kernel: it serves pointers that are not 16-byte aligned."""
        buf, y = torch.empty(x.numel() + 8, dtype=x.dtype, device="cuda"), torch.empty_like(x)
        shifted = buf[1:1 + x.numel()].view_as(x)
        shifted.copy_(x)
        assert mine.s2pk_rms_norm(p(shifted), p(w), p(y), x.shape[0], x.shape[1], EPS, None) == 0
        return y
    return torch, p, scalar_norm


def rnd(torch, *shape, seed=0):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)).bfloat16()


def same(torch, a, b):
    assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("rows,width", [(1, 2560), (3, 4096), (5, 8), (300, 2560)])
def test_norm_alone(mine, tools, rows, width):
    torch, p, scalar_norm = tools
    x, w = rnd(torch, rows, width, seed=1), rnd(torch, width, seed=2)
    y = torch.empty_like(x)
    assert mine.s2pk_rms_norm(p(x), p(w), p(y), rows, width, EPS, None) == 0
    same(torch, y, scalar_norm(x, w))


@pytest.mark.parametrize("rows", [1, 17])
def test_add_and_copy(mine, testlib, tools, rows):
    torch, p, scalar_norm = tools
    x, add, w = rnd(torch, rows, D, seed=3), rnd(torch, rows, D, seed=4), rnd(torch, D, seed=5)
    want, got, y = x.clone(), x.clone(), torch.empty_like(x)
    assert mine.s2pk_add(p(want), p(add), want.numel(), None) == 0
    assert testlib.add_norm(p(got), p(add), p(w), p(y), rows, None) == 0
    same(torch, got, want)
    same(torch, y, scalar_norm(want, w))
    assert testlib.add_norm(p(got), p(add), None, None, rows, None) == 0
    assert mine.s2pk_add(p(want), p(add), want.numel(), None) == 0
    same(torch, got, want)
    out = torch.empty_like(x)
    assert testlib.copy_norm(p(x), p(out), p(w), p(y), rows, None) == 0
    same(torch, out, x)
    same(torch, y, scalar_norm(x, w))


@pytest.mark.parametrize("rows", [1, 9])
def test_embedding_of_a_code_or_of_an_argmax(mine, testlib, tools, rows):
    torch, p, scalar_norm = tools
    table, w, logits = rnd(torch, CB, D, seed=6), rnd(torch, D, seed=7), rnd(torch, rows, CB, seed=8)
    logits[0, 7] = logits[0, 4000] = 9.0  # a tie goes to the lower index
    if rows > 1:
        logits[1] = float("nan")
        logits[2] = float("-inf")
    ids, got = (torch.empty(rows, dtype=torch.int32, device="cuda") for _ in range(2))
    assert mine.s2pk_argmax(p(logits), p(ids), rows, CB, None) == 0
    x, y = (torch.empty(rows, D, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert testlib.embed_norm(p(table), None, p(logits), p(got), p(x), p(w), p(y), rows, None) == 0
    assert torch.equal(got, ids) and int(got[0]) == 7
    same(torch, x, table[ids.long()])
    same(torch, y, scalar_norm(x, w))
    codes = torch.randint(-5, CB + 5, (rows,), dtype=torch.int32, device="cuda")
    assert testlib.embed_norm(p(table), p(codes), None, None, p(x), p(w), p(y), rows, None) == 0
    same(torch, x, table[codes.long().clamp(0, CB - 1)])
    same(torch, y, scalar_norm(x, w))
