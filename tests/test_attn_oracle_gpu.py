"""Attention of prompt rows and of decoding rows against the CPU oracle, which restates the operation order with the host's expf.

Tolerance: both sides run the same fp32 chains and round once to bf16.  What differs is expf (CUDA's and the host's are within 2 ulp)
and 1/sqrt(128) (1 ulp), an error of some 1e-6 of the sums of weights times values (of magnitude 1 to 3), so an output may at most land on the neighbouring
bf16 value - except below 1e-4, where bf16 values lie closer than that error."""
import ctypes as C

import numpy as np
import pytest

from _internal_abi import AttnArgs

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
QH, KVH, HD = 32, 8, 128


def same_or_neighbours(got, want, what):
    """bf16 bit patterns, compared on the line of ordered values"""
    order = lambda u: np.where(u & 0x8000, 0x8000 - u.astype(np.int32), u.astype(np.int32))  # noqa: E731
    far = np.abs(order(got) - order(want))
    tiny = np.maximum(np.abs((got.astype(np.uint32) << 16).view(np.float32)), np.abs((want.astype(np.uint32) << 16).view(np.float32))) < 1e-4
    assert ((far <= 1) | tiny).all(), (what, int(far.max()))
    assert (far == 0).mean() > 0.99, what


def caches(oracle_api, rng, kv8, max_seq):
    if kv8:
        kv = rng.integers(-127, 128, size=(2, KVH, max_seq, HD), dtype=np.int8)
        return kv, (rng.random((2, KVH, max_seq, 4), dtype=np.float32) * 0.02 + 0.001).astype(np.float16)
    return oracle_api.f32_to_bf16(rng.standard_normal((2, KVH, max_seq, HD), dtype=np.float32)), np.zeros((2, 1), np.float16)


@pytest.mark.parametrize("kv8", [0, 1])
@pytest.mark.parametrize("pos0,rows", [(0, 1), (0, 3), (120, 24), (300, 77), (1000, 1)])
def test_prompt_rows(testlib, oracle, kv8, pos0, rows):
    from oracle import oracle_api
    testlib.attn_single.argtypes = [C.POINTER(AttnArgs), C.c_int, C.c_void_p]
    rng, max_seq = np.random.default_rng(rows), pos0 + rows
    kv, sc = caches(oracle_api, rng, kv8, max_seq)
    q = oracle_api.f32_to_bf16(rng.standard_normal((rows, QH * HD), dtype=np.float32))
    want = np.empty_like(q)
    for r in range(rows):
        oracle.s2po_attn_single(*[oracle_api.ptr(x) for x in (q[r], kv[0], kv[1], sc[0], sc[1], want[r])], QH, KVH, pos0 + r + 1, max_seq, kv8)
    dq, dkv, dsc = (torch.from_numpy(x.view(np.int16) if x.dtype == np.uint16 else x).cuda() for x in (q, kv, sc))
    out = torch.zeros_like(dq)
    a = AttnArgs()
    a.q_heads, a.kv_heads, a.max_seq, a.kv8, a.head_dim, a.pos_row_step, a.pos0 = QH, KVH, max_seq, kv8, HD, 1, pos0
    a.kv.base0, a.kv.v_off, a.kv.sbase0, a.kv.vs_off = dkv.data_ptr(), dkv[0].nbytes, dsc.data_ptr(), dsc[0].nbytes
    a.q, a.out = dq.data_ptr(), out.data_ptr()
    assert testlib.attn_single(C.byref(a), rows, None) == 0
    torch.cuda.synchronize()
    same_or_neighbours(out.cpu().numpy().view(np.uint16), want, "prompt")


@pytest.mark.parametrize("kv8", [0, 1])
@pytest.mark.parametrize("pos", [0, 63, 64, 700])
def test_decoding_row(testlib, oracle, kv8, pos):
    from oracle import oracle_api
    testlib.attn_decode.argtypes = [C.POINTER(AttnArgs), C.c_int, C.c_void_p]
    rng, max_seq = np.random.default_rng(pos), (pos + 64) // 64 * 64
    kv, sc = caches(oracle_api, rng, kv8, max_seq)
    q = oracle_api.f32_to_bf16(rng.standard_normal((1, QH * HD), dtype=np.float32))
    want = np.empty_like(q)
    if kv8:
        oracle.s2po_attn_decode_kv8(*[oracle_api.ptr(x) for x in (q, kv[0], kv[1], sc[0], sc[1], want)], QH, KVH, pos + 1, max_seq)
    else:
        oracle.s2po_attn_decode_bf16(*[oracle_api.ptr(x) for x in (q, kv[0], kv[1], want)], QH, KVH, pos + 1, max_seq)
    dq, dkv, dsc = (torch.from_numpy(x.view(np.int16) if x.dtype == np.uint16 else x).cuda() for x in (q, kv, sc))
    out, slots = torch.zeros_like(dq), max_seq // 64
    part, ctr = torch.empty(QH * slots * 130, device="cuda"), torch.zeros(KVH, dtype=torch.int32, device="cuda")
    a = AttnArgs()
    a.q_heads, a.kv_heads, a.max_seq, a.kv8, a.head_dim, a.pos0 = QH, KVH, max_seq, kv8, HD, pos
    a.kv.base0, a.kv.v_off, a.kv.sbase0, a.kv.vs_off = dkv.data_ptr(), dkv[0].nbytes, dsc.data_ptr(), dsc[0].nbytes
    a.q, a.out, a.part, a.counters, a.n_split_slots, a.workers = dq.data_ptr(), out.data_ptr(), part.data_ptr(), ctr.data_ptr(), slots, 16
    assert testlib.attn_decode(C.byref(a), 1, None) == 0
    torch.cuda.synchronize()
    same_or_neighbours(out.cpu().numpy().view(np.uint16), want, "decode")
