"""The sum of a clip's codebook vectors, added to its rows, against the same sums in f32, rounded where the reference rounds."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
D, CB, N = 2560, 4096, 10


@pytest.mark.parametrize("rows", [1, 25, 430])
def test_rows(testlib, rows):
    g = torch.Generator(device="cuda").manual_seed(rows)
    table = (torch.randn(N * CB, D, device="cuda", generator=g) * 0.02).bfloat16()
    codes = torch.randint(-3, CB + 3, (N, rows), dtype=torch.int32, device="cuda", generator=g)  # clamped to the table
    x = torch.randn(rows + 1, D, device="cuda", generator=g).bfloat16()
    want = x.clone()
    acc = torch.zeros(rows, D, device="cuda")
    for c in range(N):
        acc = acc + table[c * CB + codes[c].long().clamp(0, CB - 1)].float()
    want[:rows] = (x[:rows].float() + acc.bfloat16().float()).bfloat16()
    testlib.vq_embed_add.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    torch.cuda.synchronize()
    assert testlib.vq_embed_add(C.c_void_p(table.data_ptr()), C.c_void_p(codes.data_ptr()), rows, C.c_void_p(x.data_ptr()), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(x.view(torch.int16), want.view(torch.int16))
