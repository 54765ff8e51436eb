"""The sum of a clip's codebook vectors, added to its rows, against the same sums in f32, rounded where the reference rounds."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
D, CB, N = 2560, 4096, 10


@pytest.mark.parametrize("rows,table_off,rows_off", [(1, 0, 0), (25, 0, 0), (430, 0, 0), (3, 1, 0), (3, 0, 1), (3, 4, 2)])  # elements past an aligned address
def test_rows(testlib, rows, table_off, rows_off):
    g = torch.Generator(device="cuda").manual_seed(rows)
    at = lambda t, off: torch.cat([t.new_zeros(off), t.flatten()])[off:].view(t.shape)  # noqa: E731
    table = at((torch.randn(N * CB, D, device="cuda", generator=g) * 0.02).bfloat16(), table_off)
    codes = torch.randint(-3, CB + 3, (N, rows), dtype=torch.int32, device="cuda", generator=g)  # clamped to the table
    x = at(torch.randn(rows + 1, D, device="cuda", generator=g).bfloat16(), rows_off)
    assert table.data_ptr() % 16 == 2 * table_off and x.data_ptr() % 16 == 2 * rows_off
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
