"""Attention that writes the units of the next wide linear, against the bf16 result packed."""
import ctypes as C

import pytest

from _internal_abi import AttnArgs, QkvPostArgs, TiledOut

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
P, I = C.c_void_p, C.c_int
QH, KVH, HD = 32, 8, 128


def p(t):
    return P(t.data_ptr())


def units(testlib, kind, rows, fill=None):
    testlib.wide_units.argtypes, testlib.wide_units.restype = [I, P, I], TiledOut
    testlib.wide_pack.argtypes = [I, P, I, I, P, P]
    lg = max(4, (rows - 1).bit_length())
    t = torch.zeros((QH * HD // 8) << lg, 8, dtype=torch.float16, device="cuda")
    return t, testlib.wide_units(kind, t.data_ptr(), rows)


def same_rows(a, b, rows):
    lg = max(4, (rows - 1).bit_length())
    view = lambda t: t.view(torch.int16).view(-1, 1 << lg, 8)[:, :rows]  # noqa: E731
    return torch.equal(view(a), view(b))


@pytest.mark.parametrize("kind", [0, 2])
@pytest.mark.parametrize("rows,kv8,pos", [(17, 1, 40), (32, 1, 700), (1, 1, 300), (130, 0, 129), (3, 0, 64)])
def test_decode_attention(testlib, kind, rows, kv8, pos):
    for f in ("attn_decode", "attn_decode_tiled"):
        getattr(testlib, f).argtypes = [C.POINTER(AttnArgs)] + ([C.POINTER(TiledOut)] if f.endswith("tiled") else []) + [I, P]
    g = torch.Generator(device="cuda").manual_seed(rows)
    max_seq = (pos + 64) // 64 * 64 + 64
    kv = torch.randint(-127, 128, (rows, 2, KVH, max_seq, HD), dtype=torch.int8, device="cuda", generator=g) if kv8 else torch.randn(rows, 2, KVH, max_seq, HD, device="cuda", generator=g).bfloat16()
    sc = (torch.rand(rows, 2, KVH, max_seq, 4, device="cuda", generator=g) * 0.02 + 0.001).half()
    q = torch.randn(rows, QH * HD, device="cuda", generator=g).bfloat16()
    out = torch.zeros_like(q)
    slots = (max_seq + 63) // 64
    part, ctr = torch.empty(rows * QH * slots * 130, device="cuda"), torch.zeros(rows * KVH, dtype=torch.int32, device="cuda")
    at = torch.randint(0, pos + 1, (rows,), dtype=torch.int32, device="cuda", generator=g)
    a = AttnArgs()
    a.q, a.out, a.q_heads, a.kv_heads, a.max_seq, a.kv8, a.head_dim = q.data_ptr(), out.data_ptr(), QH, KVH, max_seq, kv8, HD
    a.pos_arr, a.part, a.counters, a.n_split_slots, a.workers = at.data_ptr(), part.data_ptr(), ctr.data_ptr(), slots, 4
    a.kv.base0, a.kv.row_stride, a.kv.v_off = kv.data_ptr(), kv[0].nbytes, kv[0, 0].nbytes
    a.kv.sbase0, a.kv.srow_stride, a.kv.vs_off = sc.data_ptr(), sc[0].nbytes, sc[0, 0].nbytes
    want, _ = units(testlib, kind, rows)
    got, t = units(testlib, kind, rows)
    torch.cuda.synchronize()
    assert testlib.attn_decode(C.byref(a), rows, None) == 0 and testlib.wide_pack(kind, p(out), rows, QH * HD, p(want), None) == 0
    assert testlib.attn_decode_tiled_serves(C.byref(a), rows) and testlib.attn_decode_tiled(C.byref(a), C.byref(t), rows, None) == 0
    torch.cuda.synchronize()
    assert same_rows(got, want, rows) and int(ctr.abs().max()) == 0


# rows and lengths on either side of where the kernel takes one worker more: full SMs, three quarters of them, a share rounded up or by its waves
@pytest.mark.parametrize("kv8", [0, 1])
@pytest.mark.parametrize("rows,length", [(2, 1500), (3, 833), (4, 2000), (5, 4000), (7, 1800), (12, 769), (20, 2000), (28, 700), (37, 193), (42, 400), (96, 1000)])
def test_the_number_of_workers_changes_no_bit(testlib, kv8, rows, length):
    testlib.attn_decode.argtypes = [C.POINTER(AttnArgs), I, P]
    g = torch.Generator(device="cuda").manual_seed(rows)
    max_seq = (length + 63) // 64 * 64
    kv = torch.randint(-127, 128, (rows, 2, KVH, max_seq, HD), dtype=torch.int8, device="cuda", generator=g) if kv8 else torch.randn(rows, 2, KVH, max_seq, HD, device="cuda", generator=g).bfloat16()
    sc = (torch.rand(rows, 2, KVH, max_seq, 4, device="cuda", generator=g) * 0.02 + 0.001).half()
    q = torch.randn(rows, QH * HD, device="cuda", generator=g).bfloat16()
    slots = max_seq // 64
    part, ctr = torch.empty(rows * QH * slots * 130, device="cuda"), torch.zeros(rows * KVH, dtype=torch.int32, device="cuda")
    at = torch.full((rows,), length - 1, dtype=torch.int32, device="cuda")
    at[rows // 2] = 70  # a short row among them
    a = AttnArgs()
    a.q, a.q_heads, a.kv_heads, a.max_seq, a.kv8, a.head_dim = q.data_ptr(), QH, KVH, max_seq, kv8, HD
    a.pos_arr, a.part, a.counters, a.n_split_slots = at.data_ptr(), part.data_ptr(), ctr.data_ptr(), slots
    a.kv.base0, a.kv.row_stride, a.kv.v_off = kv.data_ptr(), kv[0].nbytes, kv[0, 0].nbytes
    a.kv.sbase0, a.kv.srow_stride, a.kv.vs_off = sc.data_ptr(), sc[0].nbytes, sc[0, 0].nbytes
    outs = []
    for workers in (1, max(2, min(16, 2048 // (rows * KVH)))):
        outs.append(torch.zeros_like(q))
        a.out, a.workers = outs[-1].data_ptr(), workers
        torch.cuda.synchronize()
        assert testlib.attn_decode(C.byref(a), rows, None) == 0
        torch.cuda.synchronize()
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16)) and outs[0].isfinite().all() and int(ctr.abs().max()) == 0


@pytest.mark.parametrize("kind", [0, 2])
@pytest.mark.parametrize("rows", [1, 32, 37, 38, 128])
def test_fast_attention(testlib, kind, rows):
    SEQ = 11
    testlib.fast_attn.argtypes = [C.POINTER(QkvPostArgs), P, P, I, I, P]
    testlib.fast_attn_tiled.argtypes = [C.POINTER(QkvPostArgs), P, C.POINTER(TiledOut), I, I, P]
    g = torch.Generator(device="cuda").manual_seed(rows)
    cache = torch.zeros(2, rows, 2, KVH, SEQ, HD, dtype=torch.bfloat16, device="cuda")
    out = torch.zeros(rows, QH * HD, dtype=torch.bfloat16, device="cuda")
    want, _ = units(testlib, kind, rows)
    got, t = units(testlib, kind, rows)
    for pos in range(SEQ):
        qkv = torch.randn(rows, QH + 2 * KVH, HD, device="cuda", generator=g).bfloat16()
        torch.cuda.synchronize()
        for which in (0, 1):
            a = QkvPostArgs()
            a.qkv, a.eps, a.rope_base, a.q_heads, a.kv_heads, a.max_seq, a.pos0 = qkv.data_ptr(), 1e-6, 1e6, QH, KVH, SEQ, pos
            a.kv.base0, a.kv.row_stride, a.kv.v_off = cache[which].data_ptr(), 2 * KVH * SEQ * HD * 2, KVH * SEQ * HD * 2
            if which:
                assert testlib.fast_attn_tiled(C.byref(a), None, C.byref(t), HD, rows, None) == 0
            else:
                assert testlib.fast_attn(C.byref(a), None, p(out), HD, rows, None) == 0 and testlib.wide_pack(kind, p(out), rows, QH * HD, p(want), None) == 0
        torch.cuda.synchronize()
        assert same_rows(got, want, rows), pos
        assert torch.equal(cache[0].view(torch.int16), cache[1].view(torch.int16)), pos
