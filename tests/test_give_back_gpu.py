"""A model without its resident copies of the weights: the same cache bytes and the same frames."""
import ctypes as C
import os

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
ROWS = 20  # beyond the exact-order kernels: the tick reads the f16 tiles


@pytest.mark.parametrize("int4", ["1", "0"])
def test_frames_do_not_depend_on_the_copies(testlib, synth, capi, monkeypatch, int4):
    for name, value in dict(S2P_INT8="1", S2P_INT4=int4, S2P_INT4_ALL=int4, S2P_QCACHE="0").items():
        monkeypatch.setenv(name, value)
    tl = testlib
    tl.s2p_model_give_back.argtypes = [C.c_void_p]
    ckpt = ("/dev/shm" if os.path.isdir("/dev/shm") else "/tmp") + "/s2p_synth_l2"
    synth.write_checkpoint(ckpt, n_slow=2, seed=0, generator="auto")
    runs = []
    for way in ("kept", "given back", "never made"):  # given back: the bf16 copies before the prompts, the tiles between two ticks
        monkeypatch.setenv("S2P_RESIDENT", "0" if way == "never made" else "1")
        m, give_back = C.c_void_p(), way == "given back"
        opts = capi.ModelOpts(capi.GEMM_INT8, 512, ROWS)
        capi.check(tl.s2p_model_load(ckpt.encode(), C.byref(opts), C.byref(m)), "load")
        if give_back:
            assert tl.s2p_model_give_back(m) == 1
        sessions = (C.c_void_p * ROWS)()
        for i in range(ROWS):
            cfg, s = tl.s2p_sampling_defaults(), C.c_void_p()
            cfg.temperature, cfg.seed = 0.8, 100 + i
            capi.check(tl.s2p_session_create(m, C.byref(cfg), C.byref(s)), "session")
            ids = synth.random_prompt(30 + i, 9 + i)
            capi.check(tl.s2p_session_prefill(s, ids.ctypes.data_as(C.c_void_p), None, len(ids), None, 0), "prefill")
            sessions[i] = s
        codes, eos, frames = (C.c_int32 * (10 * ROWS))(), (C.c_int * ROWS)(), []
        for tick in range(6):
            if tick == 3 and give_back:
                assert tl.s2p_model_give_back(m) == 1 and tl.s2p_model_give_back(m) == 0
            capi.check(tl.s2p_model_batch_next_frame(m, sessions, ROWS, codes, eos), "tick")
            frames.append((list(codes), list(eos)))
        if way != "kept":
            assert tl.s2p_model_give_back(m) == 0
        blob = torch.empty(int(tl.s2p_session_kv_bytes(m, 32)), dtype=torch.uint8, device="cuda")
        capi.check(tl.s2p_session_kv_save(sessions[7], 32, C.c_void_p(blob.data_ptr())), "save")
        for s in sessions:
            tl.s2p_session_destroy(s)
        tl.s2p_model_free(m)
        runs.append((frames, blob))
    for frames, blob in runs[1:]:
        assert frames == runs[0][0]
        assert torch.equal(blob, runs[0][1])
