"""Bounded waits that run out.  Every wait of the persistent tick kernel (mbarrier, flagged word, grid
barrier) has a deadline on the GPU-wide timer; past it the wait records a code, the kernel winds down
and ends normally, and the host turns the code into S2P_ERR_INTERNAL.  Here the deadline is lowered so
that this happens within microseconds: nothing hangs, traps or faults.

Uses the test twin of the library throughout (the deadline is a constant of the library image that
launches the kernels)."""
import ctypes as C
import importlib
import os

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

PIPE_ERR_TMA_WAIT, PIPE_ERR_FLAG_WAIT = 1, 3
S2P_ERR_INTERNAL = -8


def _hooks(tl):
    tl.pipe_wait_probe.restype = C.c_int
    tl.pipe_wait_probe.argtypes = [C.c_int, C.c_ulonglong, C.POINTER(C.c_int), C.POINTER(C.c_ulonglong), C.POINTER(C.c_int)]
    tl.mega_set_wait_ns.restype = C.c_int
    tl.mega_set_wait_ns.argtypes = [C.c_ulonglong]
    return tl


@pytest.mark.parametrize("which,code", [(0, PIPE_ERR_TMA_WAIT), (1, PIPE_ERR_FLAG_WAIT)])
def test_a_wait_nobody_satisfies_gives_up_at_its_deadline(testlib, which, code):
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    tl = _hooks(testlib)
    limit_ns = 200_000
    status, elapsed, got = C.c_int(0), C.c_ulonglong(0), C.c_int(1)
    assert tl.pipe_wait_probe(which, limit_ns, C.byref(status), C.byref(elapsed), C.byref(got)) == 0
    assert got.value == 0, "the wait must report failure"
    assert status.value == code
    assert limit_ns <= elapsed.value < 50 * limit_ns, elapsed.value  # gave up at the deadline, not at a poll-count backstop


def test_persistent_tick_gives_up_cleanly_and_the_model_falls_back(testlib, capi):
    """A model on the persistent tick; then the deadline drops to 100 ns, so the kernel's first wait runs
    out: that tick answers S2P_ERR_INTERNAL, the persistent path is switched off, and with the deadline
    restored the session goes on through per-stage launches."""
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    tl = _hooks(testlib)
    capi.bind(tl, capi.EXT_PROTOTYPES)
    synth = importlib.import_module("s2pro-native_b200.synth")
    os.environ.update({"S2P_INT8": "1", "S2P_INT4": "1", "S2P_INT4_ALL": "1", "S2P_QCACHE": "0", "S2P_NO_FUSED": "0", "S2P_NO_MEGA": "0"})
    ckpt = os.environ.get("S2P_TEST_CKPT_DIR", "/dev/shm") + "/s2p_synth_l2"
    synth.write_checkpoint(ckpt, n_slow=2, seed=0, generator="auto")
    opts = capi.ModelOpts(capi.GEMM_INT8, 1024, 1)
    m = C.c_void_p()
    capi.check(tl.s2p_model_load(ckpt.encode(), C.byref(opts), C.byref(m)), "load")
    cfg = tl.s2p_sampling_defaults(); cfg.temperature = 0.0
    s = C.c_void_p()
    capi.check(tl.s2p_session_create(m, C.byref(cfg), C.byref(s)), "session")
    ids = synth.random_prompt(24, 5)
    capi.check(tl.s2p_session_prefill(s, ids.ctypes.data_as(C.c_void_p), None, len(ids), None, 0), "prefill")
    codes = (C.c_int32 * 10)(); eos = C.c_int(0)
    st = capi.Stats()
    for _ in range(3):
        capi.check(tl.s2p_session_next_frame(s, codes, C.byref(eos)), "frame")
    capi.check(tl.s2p_b200_model_stats(m, C.byref(st)), "stats")
    assert st.last_tick_persistent == 1
    try:
        assert tl.mega_set_wait_ns(100) == 0
        rc = tl.s2p_session_next_frame(s, codes, C.byref(eos))
    finally:
        assert tl.mega_set_wait_ns(2_000_000_000) == 0
    assert rc == S2P_ERR_INTERNAL, rc
    torch.cuda.synchronize()  # the context is intact
    for _ in range(3):
        capi.check(tl.s2p_session_next_frame(s, codes, C.byref(eos)), "frame after the give-up")
        assert all(0 <= c < 4096 for c in codes)
    capi.check(tl.s2p_b200_model_stats(m, C.byref(st)), "stats")
    assert st.last_tick_persistent == 0, "the persistent path must stay off after a give-up"
    tl.s2p_session_destroy(s)
    tl.s2p_model_free(m)


@pytest.mark.parametrize("limit_ns", [1, 300, 900, 1500, 4000, 10000, 40000])
def test_persistent_tick_ends_wherever_its_waits_run_out(testlib, capi, limit_ns):
    """Deadlines from one poll to several stages: the tick gives up at different places, some warps of a CTA while others of it
    find what they wait for, and it always ends - with a frame or with S2P_ERR_INTERNAL - and the session goes on."""
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    tl = _hooks(testlib)
    capi.bind(tl, capi.EXT_PROTOTYPES)
    synth = importlib.import_module("s2pro-native_b200.synth")
    os.environ.update({"S2P_INT8": "1", "S2P_INT4": "1", "S2P_INT4_ALL": "1", "S2P_QCACHE": "0", "S2P_NO_FUSED": "0", "S2P_NO_MEGA": "0"})
    ckpt = os.environ.get("S2P_TEST_CKPT_DIR", "/dev/shm") + "/s2p_synth_l2"
    synth.write_checkpoint(ckpt, n_slow=2, seed=0, generator="auto")
    opts, m, s = capi.ModelOpts(capi.GEMM_INT8, 1024, 1), C.c_void_p(), C.c_void_p()
    capi.check(tl.s2p_model_load(ckpt.encode(), C.byref(opts), C.byref(m)), "load")
    cfg = tl.s2p_sampling_defaults(); cfg.temperature = 0.0
    capi.check(tl.s2p_session_create(m, C.byref(cfg), C.byref(s)), "session")
    ids = synth.random_prompt(24, 5)
    capi.check(tl.s2p_session_prefill(s, ids.ctypes.data_as(C.c_void_p), None, len(ids), None, 0), "prefill")
    codes = (C.c_int32 * 10)(); eos = C.c_int(0)
    for _ in range(2):
        capi.check(tl.s2p_session_next_frame(s, codes, C.byref(eos)), "frame")
    try:
        assert tl.mega_set_wait_ns(limit_ns) == 0
        rc = tl.s2p_session_next_frame(s, codes, C.byref(eos))
    finally:
        assert tl.mega_set_wait_ns(2_000_000_000) == 0
    assert rc in ((S2P_ERR_INTERNAL,) if limit_ns <= 300 else (0, S2P_ERR_INTERNAL)), rc
    torch.cuda.synchronize()
    for _ in range(2):
        capi.check(tl.s2p_session_next_frame(s, codes, C.byref(eos)), "frame after it")
    tl.s2p_session_destroy(s)
    tl.s2p_model_free(m)


def test_batched_tensor_core_linear_gives_up_cleanly_and_the_exact_kernel_takes_over(testlib, capi):
    """A lockstep batch of 17 sessions runs its linears on the tensor-core kernel; with that kernel's wait
    deadline at 100 ns its first wait runs out: the tick answers S2P_ERR_INTERNAL, TMEM is released, the
    status code and the arrival counters are cleared, and later ticks take the exact-order kernel."""
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    tl = _hooks(testlib)
    tl.skinny_set_wait_ns.restype = C.c_int
    tl.skinny_set_wait_ns.argtypes = [C.c_ulonglong]
    capi.bind(tl, capi.EXT_PROTOTYPES)
    synth = importlib.import_module("s2pro-native_b200.synth")
    os.environ.update({"S2P_INT8": "1", "S2P_INT4": "1", "S2P_INT4_ALL": "1", "S2P_QCACHE": "0", "S2P_NO_TC": "0"})
    ckpt = os.environ.get("S2P_TEST_CKPT_DIR", "/dev/shm") + "/s2p_synth_l2"
    synth.write_checkpoint(ckpt, n_slow=2, seed=0, generator="auto")
    n = 17
    opts = capi.ModelOpts(capi.GEMM_INT8, 256, n)
    m = C.c_void_p()
    capi.check(tl.s2p_model_load(ckpt.encode(), C.byref(opts), C.byref(m)), "load")
    sess = []
    for i in range(n):
        cfg = tl.s2p_sampling_defaults(); cfg.temperature = 0.0
        s = C.c_void_p()
        capi.check(tl.s2p_session_create(m, C.byref(cfg), C.byref(s)), "session")
        ids = synth.random_prompt(12, 40 + i)
        capi.check(tl.s2p_session_prefill(s, ids.ctypes.data_as(C.c_void_p), None, len(ids), None, 0), "prefill")
        sess.append(s)
    arr = (C.c_void_p * n)(*[s.value for s in sess])
    codes = (C.c_int32 * (10 * n))(); eos = (C.c_int * n)()
    st = capi.Stats()
    for _ in range(3):
        capi.check(tl.s2p_model_batch_next_frame(m, arr, n, codes, eos), "tick")
    capi.check(tl.s2p_b200_model_stats(m, C.byref(st)), "stats")
    kernels_tc = st.last_tick_kernels
    try:
        assert tl.skinny_set_wait_ns(100) == 0
        rc = tl.s2p_model_batch_next_frame(m, arr, n, codes, eos)
    finally:
        assert tl.skinny_set_wait_ns(2_000_000_000) == 0
    assert rc == S2P_ERR_INTERNAL, rc
    torch.cuda.synchronize()
    for _ in range(3):
        capi.check(tl.s2p_model_batch_next_frame(m, arr, n, codes, eos), "tick after the give-up")
        assert all(0 <= c < 4096 for c in codes)
    capi.check(tl.s2p_b200_model_stats(m, C.byref(st)), "stats")
    assert st.last_tick_kernels > kernels_tc, "later ticks must run the exact-order linears (more launches: 16 rows at a time)"
    for s in sess:
        tl.s2p_session_destroy(s)
    tl.s2p_model_free(m)


def _slice_waits(tl):
    tl.attn_prefill_set_wait_ns.restype = C.c_int
    tl.attn_prefill_set_wait_ns.argtypes = [C.c_ulonglong]
    return tl


def test_prompt_attention_of_a_caller_reports_a_wait_that_gave_up(testlib):
    """s2pk_attention has no synchronisation of its own: with the deadline at 1 ns a call loses rows (nearly always: a wait that the
    hardware suspends may also be satisfied before its first look at the clock), the next one says so without launching
    anything, and the one after that is whole again."""
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    tl = _slice_waits(testlib)
    rows, pos, max_seq, width = 450, 3000, 3456, 32 * 128
    g = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn(rows, width, device="cuda", generator=g).bfloat16()
    k, v = (torch.randn(8, max_seq, 128, device="cuda", generator=g).bfloat16() for _ in range(2))

    def attend():
        out = torch.full_like(q, 7.0)
        rc = tl.s2pk_attention(*[C.c_void_p(t.data_ptr()) for t in (q, k, v, out)], rows, 32, 8, 128, pos, max_seq, None)
        torch.cuda.synchronize()
        return rc, out

    rc, want = attend()
    assert rc == 0
    try:
        assert tl.attn_prefill_set_wait_ns(1) == 0
        for _ in range(100):
            rc, out = attend()
            if rc != 0:
                break
    finally:
        assert tl.attn_prefill_set_wait_ns(2_000_000_000) == 0
    assert rc == 702 and (out == 7).all()  # cudaErrorLaunchTimeout, for the call before
    rc, out = attend()
    assert rc == 0 and torch.equal(out.view(torch.int16), want.view(torch.int16))


def test_prompt_slice_whose_attention_gives_up_is_refused_and_can_be_repeated(testlib, capi):
    """A model's slice answers S2P_ERR_INTERNAL and may be sent again; neither the model nor a caller of the primitive sees the
    other's lost wait."""
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    tl = _slice_waits(_hooks(testlib))
    synth = importlib.import_module("s2pro-native_b200.synth")
    os.environ.update({"S2P_INT8": "1", "S2P_INT4": "1", "S2P_INT4_ALL": "1", "S2P_QCACHE": "0"})
    ckpt = os.environ.get("S2P_TEST_CKPT_DIR", "/dev/shm") + "/s2p_synth_l2"
    synth.write_checkpoint(ckpt, n_slow=2, seed=0, generator="auto")
    opts, m = capi.ModelOpts(capi.GEMM_INT8, 2048, 2), C.c_void_p()
    capi.check(tl.s2p_model_load(ckpt.encode(), C.byref(opts), C.byref(m)), "load")
    ids = synth.random_prompt(1500, 5)
    q = torch.zeros(64, 32 * 128, dtype=torch.bfloat16, device="cuda")
    kv = torch.zeros(8, 64, 128, dtype=torch.bfloat16, device="cuda")

    def primitive():
        args = [C.c_void_p(t.data_ptr()) for t in (q, kv, kv, q)]
        return tl.s2pk_attention(*args, 64, 32, 8, 128, 0, 64, None)

    def opened():
        cfg, s = tl.s2p_sampling_defaults(), C.c_void_p()
        cfg.temperature = 0.0
        capi.check(tl.s2p_session_create(m, C.byref(cfg), C.byref(s)), "session")
        return s

    def prefill(s):
        return tl.s2p_session_prefill(s, ids.ctypes.data_as(C.c_void_p), None, len(ids), None, 0)

    def frames(s):
        codes, eos, out = (C.c_int32 * 10)(), C.c_int(0), []
        for _ in range(3):
            capi.check(tl.s2p_session_next_frame(s, codes, C.byref(eos)), "frame")
            out.append(list(codes))
        return out

    one, two = opened(), opened()
    assert prefill(one) == 0
    want = frames(one)
    try:
        assert tl.attn_prefill_set_wait_ns(1) == 0
        for _ in range(50):
            rc = prefill(two)
            if rc != 0:
                break
            tl.s2p_session_destroy(two)
            two = opened()
    finally:
        assert tl.attn_prefill_set_wait_ns(2_000_000_000) == 0
    assert rc == S2P_ERR_INTERNAL
    assert primitive() == 0
    assert prefill(two) == 0 and frames(two) == want
    for s in (one, two):
        tl.s2p_session_destroy(s)
    tl.s2p_model_free(m)
