"""Which launches serve a frame of one session depends on the model, not on who started the process."""
import ctypes as C
import os

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("env,persistent", [({}, 0), ({"WORLD_SIZE": "8", "RANK": "3"}, 0), ({"WORLD_SIZE": "8", "S2P_NO_MEGA": "0"}, 1)])
def test_a_replica_decodes_as_a_single_process_does(mine, capi, synth, monkeypatch, env, persistent):
    for name in ("WORLD_SIZE", "RANK", "S2P_NO_MEGA", "S2P_NO_FUSED", "S2P_TICK_TRACE"):
        monkeypatch.delenv(name, raising=False)
    for name, value in dict(env, S2P_INT8="1", S2P_INT4="1", S2P_INT4_ALL="1", S2P_QCACHE="0").items():
        monkeypatch.setenv(name, value)
    ckpt = ("/dev/shm" if os.path.isdir("/dev/shm") else "/tmp") + "/s2p_synth_l2"
    synth.write_checkpoint(ckpt, n_slow=2, seed=0, generator="auto")
    opts, m, s = capi.ModelOpts(capi.GEMM_INT8, 1024, 1), C.c_void_p(), C.c_void_p()
    capi.check(mine.s2p_model_load(ckpt.encode(), C.byref(opts), C.byref(m)), "load")
    cfg = mine.s2p_sampling_defaults()
    cfg.temperature = 0.0
    capi.check(mine.s2p_session_create(m, C.byref(cfg), C.byref(s)), "session")
    ids = synth.random_prompt(24, 5)
    capi.check(mine.s2p_session_prefill(s, ids.ctypes.data_as(C.c_void_p), None, len(ids), None, 0), "prefill")
    codes, eos, st = (C.c_int32 * 10)(), C.c_int(0), capi.Stats()
    for _ in range(2):  # the second frame is the first that decodes
        capi.check(mine.s2p_session_next_frame(s, codes, C.byref(eos)), "frame")
    capi.check(mine.s2p_b200_model_stats(m, C.byref(st)), "stats")
    mine.s2p_session_destroy(s)
    mine.s2p_model_free(m)
    assert st.last_tick_persistent == persistent
