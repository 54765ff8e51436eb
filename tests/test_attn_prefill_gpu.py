"""The row-block attention of prompt slices against the single-row kernel, bit for bit."""
import ctypes as C

import pytest

from _internal_abi import AttnArgs

pytestmark = pytest.mark.gpu
QH, KVH, HD = 32, 8, 128
# which block size each of them picks is asked for in test_attn_blocks_gpu.py
SLICES = [(0, 2), (0, 129), (127, 2), (126, 5), (250, 73), (128, 128), (1000, 21), (0, 300), (40, 460), (3000, 450), (100, 50), (63, 150), (0, 209), (0, 700)]
INFINITE_VALUES = [(0, 2), (3, 3), (126, 5), (0, 24), (120, 77), (0, 300), (0, 460), (0, 40), (0, 209), (0, 700)]


@pytest.mark.parametrize("kv8", [0, 1])
@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("pos0,rows", SLICES)
def test_rows_of_a_slice_equal_single_rows(testlib, kv8, shift, pos0, rows):
    """All block sizes (their choice depends on the slice's length), ragged last blocks, tiles cut by the diagonal,
    and caches that are aligned to 4 bytes only."""
    import torch
    testlib.attn_single.argtypes = [C.POINTER(AttnArgs), C.c_int, C.c_void_p]
    g = torch.Generator(device="cuda").manual_seed(pos0 * 7 + rows)
    max_seq = (pos0 + rows + 64) // 64 * 64
    n = KVH * max_seq
    raw = torch.zeros(2 * n * HD * (1 if kv8 else 2) + 64, dtype=torch.uint8, device="cuda")
    scales = torch.full((2 * n * 4 + 32,), float("nan"), dtype=torch.float16, device="cuda")
    body = raw[shift:shift + raw.numel() - 64]
    if kv8:
        body.copy_(torch.randint(-127, 128, (2 * n * HD,), dtype=torch.int8, device="cuda", generator=g).view(torch.uint8))
        live = scales[shift // 2:shift // 2 + 2 * n * 4].view(2, KVH, max_seq, 4)
        live[:, :, :pos0 + rows] = (torch.rand(2, KVH, pos0 + rows, 4, device="cuda", generator=g) * 0.02 + 0.001).half()
    else:
        v = torch.randn(2, KVH, max_seq, HD, device="cuda", generator=g).bfloat16()
        v[:, :, pos0 + rows:] = float("nan")  # nothing past the last position may be read into a result
        body.copy_(v.flatten().view(torch.uint8))
    q = torch.randn(rows, QH * HD, device="cuda", generator=g).bfloat16()
    out, ref = torch.zeros_like(q), torch.zeros_like(q)
    a = AttnArgs()
    a.q_heads, a.kv_heads, a.max_seq, a.kv8, a.head_dim, a.pos_row_step = QH, KVH, max_seq, kv8, HD, 1
    a.kv.base0, a.kv.k_off, a.kv.v_off = raw.data_ptr() + shift, 0, n * HD * (1 if kv8 else 2)
    a.kv.sbase0, a.kv.ks_off, a.kv.vs_off = scales.data_ptr() + shift, 0, n * 8
    a.q, a.out, a.pos0 = q.data_ptr(), out.data_ptr(), pos0
    assert testlib.attn_single(C.byref(a), rows, None) == 0
    for r in range(rows):
        a.q, a.out, a.pos0 = q[r].data_ptr(), ref[r].data_ptr(), pos0 + r
        assert testlib.attn_single(C.byref(a), 1, None) == 0
    torch.cuda.synchronize()
    assert not torch.isnan(ref.float()).any()
    assert torch.equal(out.view(torch.int16), ref.view(torch.int16))


@pytest.mark.parametrize("kv8", [0, 1])
@pytest.mark.parametrize("pos0,rows", INFINITE_VALUES)
def test_infinite_values_reach_only_the_rows_that_see_them(testlib, kv8, pos0, rows):
    """Every block size: infinities and NaN in the values of the slice's second half leave the rows before it as they are."""
    import torch
    testlib.attn_single.argtypes = [C.POINTER(AttnArgs), C.c_int, C.c_void_p]
    g = torch.Generator(device="cuda").manual_seed(rows)
    max_seq, bad = pos0 + rows, pos0 + (rows + 1) // 2
    q, out, ref = (torch.randn(rows, QH * HD, device="cuda", generator=g).bfloat16() for _ in range(3))
    if kv8:  # an infinite group scale: what the quantiser makes of a vector beyond f16's range
        kv = torch.randint(1, 128, (2, KVH, max_seq, HD), dtype=torch.int8, device="cuda", generator=g)
        sc = (torch.rand(2, KVH, max_seq, 4, device="cuda", generator=g) * 0.02 + 0.001).half()
        sc[1, :, bad:, ::2], sc[1, :, bad:, 1::2] = float("inf"), float("nan")
    else:
        kv = torch.randn(2, KVH, max_seq, HD, device="cuda", generator=g).bfloat16()
        kv[1, :, bad:, ::2], kv[1, :, bad:, 1::2] = float("inf"), float("nan")
        sc = kv
    a = AttnArgs()
    a.q_heads, a.kv_heads, a.max_seq, a.kv8, a.head_dim, a.pos_row_step = QH, KVH, max_seq, kv8, HD, 1
    a.kv.base0, a.kv.v_off, a.kv.sbase0, a.kv.vs_off = kv.data_ptr(), kv[0].nbytes, sc.data_ptr(), sc[0].nbytes
    a.q, a.out, a.pos0 = q.data_ptr(), out.data_ptr(), pos0
    assert testlib.attn_single(C.byref(a), rows, None) == 0
    for r in range(rows):
        a.q, a.out, a.pos0 = q[r].data_ptr(), ref[r].data_ptr(), pos0 + r
        assert testlib.attn_single(C.byref(a), 1, None) == 0
    torch.cuda.synchronize()
    seen = bad - pos0
    assert ref[:seen].isfinite().all() and not ref[seen:].isfinite().any()
    assert torch.equal(out[:seen].view(torch.int16), ref[:seen].view(torch.int16))
    assert torch.equal(out.isnan(), ref.isnan()) and torch.equal(out.isinf(), ref.isinf())
