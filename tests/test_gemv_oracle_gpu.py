"""The exact-order linear against the CPU oracle, bit for bit: every batch size it serves, both weight formats and grouped INT8, tiles of
K whole to a warp and shared by a CTA's warps, ragged rows."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
G = 32


def p(t):
    return C.c_void_p(t.data_ptr())


def against_the_oracle(mine, oracle, kind, n, k, batches):
    from oracle import oracle_api
    most = max(batches)
    rng = np.random.default_rng(n)
    w = rng.integers(0, 256, size=(n, k // 2 if kind == "int4" else k), dtype=np.uint8)
    s = rng.random((n, 1 if kind == "int8" else k // G), dtype=np.float32) * 0.01 + 0.001
    s = s if kind == "int8" else s.astype(np.float16)
    x = oracle_api.f32_to_bf16(rng.standard_normal((most, k), dtype=np.float32))
    want = np.empty((most, n), np.uint16)
    args = [oracle_api.ptr(a) for a in (want, x, w, s)] + [most, n, k]
    if kind == "int8":
        oracle.s2po_gemv_int8(*args)
    else:
        (oracle.s2po_gemv_g if kind == "int8_grouped" else oracle.s2po_gemv_p)(*args, G)
    dw, ds, dx = (torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a).cuda() for a in (w, s, x))
    for rows in batches:
        y = torch.full((rows + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
        args = [p(y), p(dx), p(dw), p(ds), rows, n, k]
        if kind == "int8":
            assert mine.s2p_int8_gemv(*args, None) == 0
        else:
            assert (mine.s2p_intq_gemv if kind == "int8_grouped" else mine.s2p_int4p_gemv)(*args, G, None) == 0
        got = y.view(torch.int16).cpu().numpy().view(np.uint16)
        assert np.array_equal(got[:rows], want[:rows]), rows
        assert (got[rows] == oracle_api.f32_to_bf16(np.float32([7.0]))[0]).all()


@pytest.mark.parametrize("kind", ["int8", "int8_grouped", "int4"])
@pytest.mark.parametrize("n,k,all_rows", [(37, 512, True), (1029, 4608, True), (6145, 1024, True), (14209, 512, False), (19457, 512, False)])
def test_every_batch_size_gives_the_oracles_bits(mine, oracle, kind, n, k, all_rows):
    against_the_oracle(mine, oracle, kind, n, k, range(1, 17) if all_rows else (1, 2))  # many rows of weights: what differs is the one-row kernel


# either side of where a CTA's warps stop sharing rows (148 SMs x 5 or 6 CTAs x 4 rows; 12 tiles of K) and of two warps to a scheduler
@pytest.mark.parametrize("kind", ["int8", "int8_grouped", "int4"])
@pytest.mark.parametrize("n,k", [(2960, 512), (2961, 1024), (3552, 512), (3553, 1024), (1029, 6144), (1029, 6656), (4732, 512), (4733, 1024)])
def test_both_sides_of_a_rule_give_the_oracles_bits(mine, oracle, kind, n, k):
    against_the_oracle(mine, oracle, kind, n, k, (1, 2, 3, 4, 5, 9))


# a tile or two of K; three rows up to twelve tiles; two rows where some SMs get a fourth CTA; five to eight rows up to two waves of shared rows; eight tiles of K, up to 12 and 17 SMs' worth of quads
@pytest.mark.parametrize("kind", ["int8", "int8_grouped", "int4"])
@pytest.mark.parametrize("n,k,batches", [(2559, 512, (1, 2, 3, 8)), (4095, 1024, (1, 2, 3, 4, 8)), (2961, 1536, (1, 3)), (2961, 6144, (3,)), (2961, 6656, (3,)), (4736, 2560, (5, 8)), (4737, 2560, (5, 8)),
                                         (5920, 2560, (6,)), (5921, 2560, (6,)), (7104, 4096, (1, 2)), (7105, 4096, (1,)), (7104, 512, (2,)), (7105, 1536, (2,)), (9472, 1536, (2,)), (9473, 1536, (2,)), (10064, 4096, (2, 7)), (10065, 4096, (2, 7))])
def test_both_sides_of_the_rules_on_tiles_give_the_oracles_bits(mine, oracle, kind, n, k, batches):
    against_the_oracle(mine, oracle, kind, n, k, batches)
