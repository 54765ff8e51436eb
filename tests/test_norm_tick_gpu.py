"""The add and norm of a tick's rows and of a slice's, either side of where the kernels change, against the separate element-wise ones."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
D = 2560


def p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("rows", [1, 2, 255, 256, 257, 700])
def test_add_and_norm(mine, testlib, rows):
    testlib.add_norm_to.argtypes = [C.c_void_p] * 5 + [C.c_int, C.c_void_p]
    g = torch.Generator(device="cuda").manual_seed(rows)
    src, add = (torch.randn(rows, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    gain = torch.randn(D, device="cuda", generator=g).bfloat16()
    buf, want = torch.empty(rows * D + 8, dtype=torch.bfloat16, device="cuda"), torch.empty_like(src)
    total = buf[1:1 + rows * D].view(rows, D)  # not 16-byte aligned: the element-wise norm
    total.copy_(src)
    assert mine.s2pk_add(p(total), p(add), total.numel(), None) == 0
    assert mine.s2pk_rms_norm(p(total), p(gain), p(want), rows, D, 1e-6, None) == 0
    x, y = torch.empty_like(src), torch.full((rows + 1, D), 7.0, dtype=torch.bfloat16, device="cuda")
    assert testlib.add_norm_to(p(src), p(add), p(x), p(gain), p(y), rows, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(x.view(torch.int16), total.view(torch.int16))
    assert torch.equal(y[:rows].view(torch.int16), want.view(torch.int16)) and (y[rows] == 7).all()
