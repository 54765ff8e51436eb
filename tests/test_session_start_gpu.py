"""What happens around a request's first frame: sessions on recycled device memory."""
import ctypes as C
import os

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def model(mine, capi, synth):
    saved = {k: os.environ.get(k) for k in ("S2P_INT8", "S2P_INT4", "S2P_INT4_ALL", "S2P_QCACHE")}
    os.environ.update(S2P_INT8="1", S2P_INT4="1", S2P_INT4_ALL="1", S2P_QCACHE="0")
    ckpt = ("/dev/shm" if os.path.isdir("/dev/shm") else "/tmp") + "/s2p_synth_l2"
    synth.write_checkpoint(ckpt, n_slow=2, seed=0, generator="auto")
    opts, m = capi.ModelOpts(capi.GEMM_INT8, 1024, 4), C.c_void_p()
    capi.check(mine.s2p_model_load(ckpt.encode(), C.byref(opts), C.byref(m)), "load")
    yield m
    mine.s2p_model_free(m)
    for k, v in saved.items():
        os.environ.pop(k) if v is None else os.environ.__setitem__(k, v)


def opened(mine, capi, m, temperature=0.0, seed=1):
    cfg = mine.s2p_sampling_defaults()
    cfg.temperature, cfg.seed = temperature, seed
    s = C.c_void_p()
    capi.check(mine.s2p_session_create(m, C.byref(cfg), C.byref(s)), "create")
    return s


def frames(mine, capi, s, ids, n):
    capi.check(mine.s2p_session_prefill(s, ids.ctypes.data_as(C.c_void_p), None, len(ids), None, 0), "prefill")
    out, codes, eos = [], (C.c_int32 * 10)(), C.c_int(0)
    for _ in range(n):
        capi.check(mine.s2p_session_next_frame(s, codes, C.byref(eos)), "frame")
        out.append((list(codes), eos.value))
    return out


def test_a_recycled_session_is_a_fresh_one(mine, capi, synth, model):
    """Sessions are opened on memory that others left behind, in another order and after longer contexts."""
    ids = synth.random_prompt(40, 3)
    first = opened(mine, capi, model)
    want = frames(mine, capi, first, ids, 4)
    others = [opened(mine, capi, model, 0.8, 5 + i) for i in range(3)]
    for o in others:
        frames(mine, capi, o, synth.random_prompt(300, 9), 3)
    for s in (others[1], first, others[0], others[2]):
        mine.s2p_session_destroy(s)
    again = [opened(mine, capi, model) for _ in range(4)]
    assert len({s.value for s in again}) == 4
    for s in again:
        assert frames(mine, capi, s, ids, 4) == want
    full = C.c_void_p()
    cfg = mine.s2p_sampling_defaults()
    assert mine.s2p_session_create(model, C.byref(cfg), C.byref(full)) == -9, "the session limit does not count pooled memory"
    for s in again:
        mine.s2p_session_destroy(s)
