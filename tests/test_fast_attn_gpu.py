"""The fast stack's rotation, cache append and attention in one kernel against the two it stands for, pass after pass."""
import ctypes as C

import pytest

from _internal_abi import AttnArgs, QkvPostArgs

pytestmark = pytest.mark.gpu
QH, KVH, HD, SEQ = 32, 8, 128, 16


@pytest.mark.parametrize("rows", [1, 3, 130])
@pytest.mark.parametrize("with_norm", [True, False])
def test_passes_equal_the_two_kernels(testlib, rows, with_norm):
    import torch
    P, I = C.c_void_p, C.c_int
    testlib.fast_attn.argtypes = [C.POINTER(QkvPostArgs), P, P, I, I, P]
    testlib.qkv_post.argtypes, testlib.attn_single.argtypes = [C.POINTER(QkvPostArgs), I, P], [C.POINTER(AttnArgs), I, P]
    g = torch.Generator(device="cuda").manual_seed(rows)
    cache = torch.full((2, rows, 2, KVH, SEQ, HD), float("nan"), dtype=torch.bfloat16, device="cuda")  # what is not written must not be read
    gain = (1 + 0.1 * torch.randn(HD, device="cuda", generator=g)).bfloat16()
    q, got, want = (torch.zeros(rows, QH * HD, dtype=torch.bfloat16, device="cuda") for _ in range(3))
    for pos in range(SEQ):
        qkv = torch.randn(rows, QH + 2 * KVH, HD, device="cuda", generator=g).bfloat16()
        torch.cuda.synchronize()
        for which in (0, 1):
            a = QkvPostArgs()
            a.qkv, a.q, a.eps, a.rope_base = qkv.data_ptr(), q.data_ptr(), 1e-6, 1e6
            a.q_norm = a.k_norm = gain.data_ptr() if with_norm else None
            a.q_heads, a.kv_heads, a.max_seq, a.pos0 = QH, KVH, SEQ, pos
            a.kv.base0, a.kv.row_stride, a.kv.v_off = cache[which].data_ptr(), 2 * KVH * SEQ * HD * 2, KVH * SEQ * HD * 2
            if which == 0:
                assert testlib.fast_attn(C.byref(a), None, got.data_ptr(), HD, rows, None) == 0
                continue
            assert testlib.qkv_post(C.byref(a), rows, None) == 0
            b = AttnArgs()
            b.q, b.out, b.q_heads, b.kv_heads, b.max_seq, b.head_dim, b.pos0, b.kv = q.data_ptr(), want.data_ptr(), QH, KVH, SEQ, HD, pos, a.kv
            assert testlib.attn_single(C.byref(b), rows, None) == 0
        torch.cuda.synchronize()
        assert torch.equal(got.view(torch.int16), want.view(torch.int16)), pos
        assert torch.equal(cache[0].view(torch.int16), cache[1].view(torch.int16)), pos
