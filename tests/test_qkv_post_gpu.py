"""Split, head norm, RoPE and cache append in one kernel against the contract launchers that do one step each."""
import ctypes as C

import pytest

from _internal_abi import QkvPostArgs

pytestmark = pytest.mark.gpu
QH, KVH, HD, EPS, BASE = 32, 8, 128, 1e-6, 1e6


@pytest.mark.parametrize("with_norm", [True, False])
@pytest.mark.parametrize("rows,pos0", [(1, 0), (1, 8190), (5, 1021), (130, 37)])
def test_rows_equal_the_separate_steps(mine, testlib, rows, pos0, with_norm):
    import torch
    testlib.qkv_post.argtypes = [C.POINTER(QkvPostArgs), C.c_int, C.c_void_p]
    p = lambda t: C.cast(C.c_void_p(t.data_ptr()), C.c_void_p)  # noqa: E731
    g = torch.Generator(device="cuda").manual_seed(rows)
    max_seq = pos0 + rows + 3
    qkv = torch.randn(rows, QH + 2 * KVH, HD, device="cuda", generator=g).bfloat16()
    gain = (1 + 0.1 * torch.randn(HD, device="cuda", generator=g)).bfloat16()
    q, k, v = (t.clone(memory_format=torch.contiguous_format) for t in qkv.split([QH, KVH, KVH], 1))
    cache, out = torch.zeros(2, 2, KVH, max_seq, HD, dtype=torch.bfloat16, device="cuda"), torch.zeros_like(q)
    if with_norm:
        assert mine.s2pk_qk_norm(p(q), p(gain), rows, QH, HD, EPS, None) == 0
        assert mine.s2pk_qk_norm(p(k), p(gain), rows, KVH, HD, EPS, None) == 0
    assert mine.s2pk_rope(p(q), p(k), rows, QH, KVH, HD, pos0, BASE, None) == 0
    assert mine.s2pk_kv_append(p(k), p(v), p(cache[0, 0]), p(cache[0, 1]), rows, KVH, HD, pos0, max_seq, None) == 0
    a = QkvPostArgs()
    a.qkv, a.q, a.eps, a.rope_base = qkv.data_ptr(), out.data_ptr(), EPS, BASE
    a.q_norm = a.k_norm = gain.data_ptr() if with_norm else None
    a.q_heads, a.kv_heads, a.max_seq, a.pos0, a.pos_row_step = QH, KVH, max_seq, pos0, 1
    a.kv.base0, a.kv.v_off = cache[1].data_ptr(), KVH * max_seq * HD * 2
    assert testlib.qkv_post(C.byref(a), rows, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int16), q.view(torch.int16))
    assert torch.equal(cache[1].view(torch.int16), cache[0].view(torch.int16))
    # INT8 cache: one f16 scale per 32 elements, codes rounded to nearest
    codes = torch.zeros(2, KVH, max_seq, HD, dtype=torch.int8, device="cuda")
    scales = torch.zeros(2, KVH, max_seq, 4, dtype=torch.float16, device="cuda")
    a.kv8, a.kv.base0, a.kv.v_off, a.kv.sbase0, a.kv.vs_off = 1, codes.data_ptr(), KVH * max_seq * HD, scales.data_ptr(), KVH * max_seq * 8
    assert testlib.qkv_post(C.byref(a), rows, None) == 0
    x = cache[0][:, :, pos0:pos0 + rows].float().reshape(2, KVH, rows, 4, 32)
    sc = (x.abs().amax(-1) / 127).half()
    assert torch.equal(scales[:, :, pos0:pos0 + rows], sc)
    want = (x / sc.float()[..., None]).round().clamp(-127, 127).to(torch.int8).reshape(2, KVH, rows, HD)
    assert torch.equal(codes[:, :, pos0:pos0 + rows], want)
