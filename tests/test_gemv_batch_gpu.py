"""Rows of a small batch against the same rows one at a time: the same bits whatever the batch, the split or the matrix's edges."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("rows", [2, 3, 5, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(1, 512), (1029, 1536), (1029, 4608), (2561, 4096), (6145, 1024)])  # whole and shared tile turns, ragged rows
def test_batch_rows_equal_single_rows(mine, kind, rows, n, k):
    g = torch.Generator(device="cuda").manual_seed(rows)
    w = torch.randint(0, 256, (n, k // 2 if kind == 2 else k), dtype=torch.uint8, device="cuda", generator=g)
    s = torch.rand(n, 1 if kind == 0 else k // 32, device="cuda", generator=g) * 0.01 + 0.001
    s = s if kind == 0 else s.half()
    x = torch.randn(rows, k, device="cuda", generator=g).bfloat16()
    got = torch.full((rows + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
    want = torch.empty((rows, n), dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()

    def gemv(y, a, m):
        if kind == 0:
            return mine.s2p_int8_gemv(p(y), p(a), p(w), p(s), m, n, k, None)
        return (mine.s2p_intq_gemv if kind == 1 else mine.s2p_int4p_gemv)(p(y), p(a), p(w), p(s), m, n, k, 32, None)

    assert gemv(got, x, rows) == 0
    for r in range(rows):
        assert gemv(want[r], x[r], 1) == 0
    torch.cuda.synchronize()
    assert torch.equal(got[:rows].view(torch.int16), want.view(torch.int16))
    assert (got[rows] == 7).all()
