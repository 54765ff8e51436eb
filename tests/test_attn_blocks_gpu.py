"""Prompt attention behind a context, slices whose length picks each block size in turn, against single rows, bit for bit."""
import ctypes as C

import pytest

import test_attn_prefill_gpu as slices
from _internal_abi import AttnArgs

pytestmark = pytest.mark.gpu
QH, KVH, HD = 32, 8, 128


POS0, LENGTHS = 1003, [2, 37, 72, 73, 108, 109, 143, 144, 145, 210, 250, 280, 430]


@pytest.mark.parametrize("calls", [[(POS0, n) for n in LENGTHS], slices.SLICES, slices.INFINITE_VALUES], ids=["behind a context", "slices", "infinite values"])
def test_every_block_size_is_reached(testlib, calls):
    """By the slices of the tests that claim it: which length picks which size is an estimate of times, and changes with them."""
    testlib.attn_prefill_rows_of_block.argtypes = [C.POINTER(AttnArgs), C.c_int]
    sizes = set()
    for pos0, rows in calls:
        a = AttnArgs()
        a.q_heads, a.kv_heads, a.head_dim, a.pos_row_step, a.pos0 = QH, KVH, HD, 1, pos0
        sizes.add(testlib.attn_prefill_rows_of_block(C.byref(a), rows))
    assert sizes == {2, 4, 6, 8, 12, 16, 24}


@pytest.mark.parametrize("kv8", [0, 1])
@pytest.mark.parametrize("rows", LENGTHS)
def test_rows_equal_single_rows(testlib, kv8, rows):
    import torch
    testlib.attn_single.argtypes = [C.POINTER(AttnArgs), C.c_int, C.c_void_p]
    g = torch.Generator(device="cuda").manual_seed(rows)
    pos0 = POS0
    max_seq = pos0 + rows
    kv = torch.randint(-127, 128, (2, KVH, max_seq, HD), dtype=torch.int8, device="cuda", generator=g) if kv8 else torch.randn(2, KVH, max_seq, HD, device="cuda", generator=g).bfloat16()
    sc = (torch.rand(2, KVH, max_seq, 4, device="cuda", generator=g) * 0.02 + 0.001).half()
    q = torch.randn(rows, QH * HD, device="cuda", generator=g).bfloat16()
    out, ref = torch.zeros_like(q), torch.zeros_like(q)
    a = AttnArgs()
    a.q_heads, a.kv_heads, a.max_seq, a.kv8, a.head_dim, a.pos_row_step = QH, KVH, max_seq, kv8, HD, 1
    a.kv.base0, a.kv.v_off, a.kv.sbase0, a.kv.vs_off = kv.data_ptr(), kv[0].nbytes, sc.data_ptr(), sc[0].nbytes
    a.q, a.out, a.pos0 = q.data_ptr(), out.data_ptr(), pos0
    assert testlib.attn_single(C.byref(a), rows, None) == 0
    for r in range(rows):
        a.q, a.out, a.pos0 = q[r].data_ptr(), ref[r].data_ptr(), pos0 + r
        assert testlib.attn_single(C.byref(a), 1, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int16), ref.view(torch.int16))
