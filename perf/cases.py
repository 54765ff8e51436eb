"""The work a user of this library has it do, as cases that can be timed.

Three kinds of pass, each through the C ABI that `s2pro-native_b200/capi.py` binds:

  decode  one lockstep frame (s2p_model_batch_next_frame) of `rows` sessions that already hold about
          `context` cached positions each: what a server does 21 times a second for every listener.  A
          session that ended is replaced before the next pass, as a server does.
  start   one request up to its first frame: session, cached voice prefix if there is one (kv_load), prompt
          in slices of at most 2048 tokens with a reference clip's codes injected if there is one,
          the prompt's cache kept for the next request (kv_save), first frame, session closed.
  linear  one s2p_linear_forward, for callers that build their own layers from the library's linears.

The model is the full one (36 backbone layers, 4 fast layers) on a seeded random checkpoint.  It is loaded once
per option set and process, as a server would; the seed of a case changes prompts, contexts and samplers.
"""
import ctypes as C
import importlib
import math
import os
import random
import shutil

import numpy as np
import torch

_capi = importlib.import_module("s2pro-native_b200.capi")
_synth = importlib.import_module("s2pro-native_b200.synth")

LAYERS, FAST_LAYERS, CODEBOOKS = 36, 4, 10
DIM, QKV, Q_WIDTH, FFN = 2560, 6144, 4096, 9728
SEMANTIC_FIRST, SEMANTIC_COUNT = 151678, 4096
HEAD_ROWS = 4097
LAYER_SHAPES = ((QKV, DIM), (DIM, Q_WIDTH), (2 * FFN, DIM), (DIM, FFN))
LAYER_WEIGHTS = sum(n * k for n, k in LAYER_SHAPES)
LAYER_ROWS = sum(n for n, _ in LAYER_SHAPES)
SLICE = 2048                     # tokens one prefill call takes
CACHE_LIMIT = 24e9               # bytes of KV cache one state may hold (three of them are in memory at a time)
CONTEXT_SIZES = (2048, 4096, 9216)
SESSIONS = 256


def listed():
    return [
        # a caller's own layer at batch 1: one call, where the launch and the first bytes count
        {"name": "linear_1row", "kind": "linear", "weights": "int4", "n": 2 * FFN, "k": DIM, "rows": 1},
        # one listener, the default configuration and the headline of the benchmark
        {"name": "frame_int4", "kind": "decode", "weights": "int4", "kv": "int8", "rows": 1, "context": 512, "temperature": 0.8},
        # the same with 8-bit weights, greedy
        {"name": "frame_int8", "kind": "decode", "weights": "int8", "kv": "int8", "rows": 1, "context": 300, "temperature": 0.0},
        # one listener deep in a long read
        {"name": "frame_int4_long", "kind": "decode", "weights": "int4", "kv": "int8", "rows": 1, "context": 8000, "temperature": 0.8},
        # a few listeners, an odd count
        {"name": "batch3_int4", "kind": "decode", "weights": "int4", "kv": "int8", "rows": 3, "context": 700, "temperature": 0.8},
        {"name": "batch8_int4", "kind": "decode", "weights": "int4", "kv": "int8", "rows": 8, "context": 1024, "temperature": 0.8},
        # the largest exact-order batch, with 8-bit weights and an unquantised cache
        {"name": "batch16_int8_kvbf16", "kind": "decode", "weights": "int8", "kv": "bf16", "rows": 16, "context": 1500, "temperature": 0.8},
        # a server with long contexts
        {"name": "batch32_int4_8k", "kind": "decode", "weights": "int4", "kv": "int8", "rows": 32, "context": 8192, "temperature": 0.8},
        # a full server with short ones
        {"name": "batch128_int4", "kind": "decode", "weights": "int4", "kv": "int8", "rows": 128, "context": 1024, "temperature": 0.8},
        # a request that finds its voice in the prefix cache, with a short sentence and a clip tail of its own
        {"name": "start_cached_voice", "kind": "start", "weights": "int4", "kv": "int8", "prefix": 1024, "prompt": 77, "clip": 25},
        # a request with a paragraph, nothing cached
        {"name": "start_512", "kind": "start", "weights": "int4", "kv": "int8", "prefix": 0, "prompt": 512, "clip": 0},
        # a request with a long document and a clip
        {"name": "start_8k", "kind": "start", "weights": "int4", "kv": "int8", "prefix": 0, "prompt": 8100, "clip": 430},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    weights = rng.choice(("int4", "int4", "int8"))
    kv = rng.choice(("int8", "int8", "int8", "bf16"))
    kind = rng.choice(("decode", "decode", "decode", "start", "start", "linear"))
    if kind == "linear":
        n, k = rng.choice(LAYER_SHAPES)
        return {"kind": kind, "weights": weights, "n": n, "k": k, "rows": _spread(rng, 1, 2048)}
    if kind == "start":
        prompt = _spread(rng, 3, 8100)
        prefix = _spread(rng, 16, 2048) if prompt < 2048 and rng.random() < 0.5 else 0
        clip = rng.randrange(1, prompt // 3 + 1) if rng.random() < 0.5 else 0
        return {"kind": kind, "weights": weights, "kv": kv, "prefix": prefix, "prompt": prompt, "clip": clip}
    context = _spread(rng, 64, 8192)
    most = int(CACHE_LIMIT / (_context_size(context) * _kv_bytes(kv)))
    return {"kind": kind, "weights": weights, "kv": kv, "rows": _spread(rng, 1, max(1, min(128, most))), "context": context,
            "temperature": rng.choice((0.8, 0.8, 0.0))}


def work(case):
    """Every weight, cache byte and activation once; the fast stack's arithmetic is done once per codebook."""
    if case["kind"] == "linear":
        n, k, m = case["n"], case["k"], case["rows"]
        return {"bytes": _weight_bytes(case["weights"], n * k, n) + 2 * m * (n + k), "flops": 2 * n * k * m}
    layer = _weight_bytes(case["weights"], LAYER_WEIGHTS, LAYER_ROWS)
    model = (LAYERS + FAST_LAYERS) * layer + _weight_bytes(case["weights"], 4096 * DIM, 4096) + HEAD_ROWS * (DIM + 4)
    fast_flops = 2 * (CODEBOOKS * FAST_LAYERS * LAYER_WEIGHTS + (CODEBOOKS - 1) * 4096 * DIM + HEAD_ROWS * DIM)
    per_position = 4 * Q_WIDTH * LAYERS  # query x key and weight x value of one (row, position) pair, all layers
    kv = _kv_bytes(case["kv"])
    if case["kind"] == "decode":
        rows, cached = case["rows"], case["rows"] * _mean_context(case)
        return {"bytes": model + kv * (cached + rows), "flops": rows * (2 * LAYERS * LAYER_WEIGHTS + fast_flops) + per_position * cached}
    p, c = case["prompt"], case["prefix"]
    return {"bytes": model + kv * (2 * c + 2 * p + (c + p)), "flops": 2 * p * LAYERS * LAYER_WEIGHTS + fast_flops + per_position * (p * c + p * (p + 1) // 2)}


def tolerance(case):
    # frames are token ids and caches are bytes: they come out the same or they are wrong
    return {"rel": 1e-2} if case["kind"] == "linear" else "exact"


def prepare(case, seed):
    torch.cuda.set_device(0)
    state = {"linear": _Layer, "decode": _Lockstep, "start": _Request}[case["kind"]](case, seed)
    torch.cuda.synchronize()
    return state


def run(state):
    return state.run()


# ---- sizes ---------------------------------------------------------------------------------------------------

def _weight_bytes(weights, count, rows):
    """4-bit codes with an f16 scale per 32 of them, or 8-bit codes with an f32 scale per row."""
    return count // 2 + count // 32 * 2 if weights == "int4" else count + 4 * rows


def _kv_bytes(kv):
    """Cache bytes of one position over all layers: 16 vectors of 128, 8-bit ones with an f16 scale per 32."""
    return LAYERS * 16 * (128 + 8 if kv == "int8" else 256)


def _context_size(tokens):
    return next(c for c in CONTEXT_SIZES if c >= tokens + min(512, tokens))


def _own_most(case):
    return max(1, min(256, case["context"] // 4))


def _mean_context(case):
    return case["context"] - _own_most(case) // 2


# ---- the model and its sessions ------------------------------------------------------------------------------

def _checkpoint():
    for base in ("/dev/shm", "/tmp"):
        path = os.path.join(base, "s2p_perf_l%d_%d" % (LAYERS, os.getuid()))
        if os.path.exists(os.path.join(path, "synth.json")) or (os.access(base, os.W_OK) and shutil.disk_usage(base).free > 12e9):
            break
    _synth.write_checkpoint(path, n_slow=LAYERS, seed=1, generator="cuda")
    return path


class _Engine:
    """One loaded model; `free` counts the sessions it can still open."""
    loaded = []

    def __init__(self, key):
        weights, kv, ctx_len = self.key = key
        int4 = "1" if weights == "int4" else "0"
        os.environ.update(S2P_INT8="1", S2P_INT4=int4, S2P_INT4_ALL=int4, S2P_KV8="1" if kv == "int8" else "0", S2P_QCACHE="0")
        self.lib, self.free, self.m = _capi.lib(), SESSIONS, C.c_void_p()
        opts = _capi.ModelOpts(_capi.GEMM_INT8, ctx_len, SESSIONS)
        _capi.check(self.lib.s2p_model_load(_checkpoint().encode(), C.byref(opts), C.byref(self.m)), "s2p_model_load")

    @classmethod
    def of(cls, weights, kv, ctx_len, sessions):
        key = (weights, kv, ctx_len)
        for e in cls.loaded:
            if e.key == key and e.free >= sessions:
                cls.loaded.remove(e)
                break
        else:
            for e in [e for e in cls.loaded if e.free == SESSIONS][: max(0, len(cls.loaded) - 3)]:
                cls.loaded.remove(e)
                e.lib.s2p_model_free(e.m)
            e = cls(key)
        cls.loaded.append(e)
        return e


class _Session:
    def __init__(self, engine, temperature, seed):
        self.engine, self.h = engine, C.c_void_p()
        cfg = engine.lib.s2p_sampling_defaults()
        cfg.temperature, cfg.top_p, cfg.seed = temperature, 0.8, seed
        _capi.check(engine.lib.s2p_session_create(engine.m, C.byref(cfg), C.byref(self.h)), "s2p_session_create")
        engine.free -= 1

    def close(self):
        if self.h:
            self.engine.lib.s2p_session_destroy(self.h)
            self.h = C.c_void_p()
            self.engine.free += 1

    __del__ = close

    def load(self, blob, tokens):
        _capi.check(self.engine.lib.s2p_session_kv_load(self.h, C.c_void_p(blob.data_ptr()), tokens), "s2p_session_kv_load")

    def save(self, blob, tokens):
        _capi.check(self.engine.lib.s2p_session_kv_save(self.h, tokens, C.c_void_p(blob.data_ptr())), "s2p_session_kv_save")

    def prefill(self, ids, mask=None, part=None):
        m = mask.ctypes.data_as(C.c_void_p) if part else None
        _capi.check(self.engine.lib.s2p_session_prefill(self.h, ids.ctypes.data_as(C.c_void_p), m, len(ids), C.byref(part) if part else None,
                                                        1 if part else 0), "s2p_session_prefill")


def _blob(engine, tokens):
    return torch.empty(int(engine.lib.s2p_session_kv_bytes(engine.m, tokens)), dtype=torch.uint8, device="cuda")


def _saved_prefix(engine, ids):
    s = _Session(engine, 0.0, 1)
    for lo in range(0, len(ids), SLICE):
        s.prefill(ids[lo:lo + SLICE])
    blob = _blob(engine, len(ids))
    s.save(blob, len(ids))
    s.close()
    return blob


class _Lockstep:
    """Sessions past their first frames.  They share most of their context (one voice) and differ in the rest, so
    the lengths are ragged."""

    def __init__(self, case, seed):
        rng = random.Random(seed)
        n, self.shared = case["rows"], case["context"] - _own_most(case)
        self.engine = _Engine.of(case["weights"], case["kv"], _context_size(case["context"]), n + 1)
        self.blob = _saved_prefix(self.engine, _synth.random_prompt(self.shared, seed))
        self.temperature, self.next_seed = case["temperature"], 1 + (seed % 1000003) * 1000
        self.own = [_synth.random_prompt(rng.randrange(1, _own_most(case) + 1), seed * 131 + 7 + i) for i in range(n)]
        self.sessions = [self.opened(i) for i in range(n)]
        self.codes, self.eos = np.zeros((n, CODEBOOKS), np.int32), np.zeros(n, np.int32)
        self.handles = (C.c_void_p * n)(*[s.h for s in self.sessions])
        for _ in range(2):  # the first frame comes from the prompt, the second is the first of the steady ones
            self.run()

    def opened(self, i):
        self.next_seed += 1
        s = _Session(self.engine, self.temperature, self.next_seed)
        s.load(self.blob, self.shared)
        s.prefill(self.own[i])
        return s

    def run(self):
        for i in np.nonzero(self.eos)[0]:
            self.sessions[i].close()
            self.sessions[i] = self.opened(i)
            self.handles[i] = self.sessions[i].h
        e = self.engine
        _capi.check(e.lib.s2p_model_batch_next_frame(e.m, self.handles, len(self.sessions), self.codes.ctypes.data_as(C.POINTER(C.c_int32)),
                                                     self.eos.ctypes.data_as(C.POINTER(C.c_int))), "s2p_model_batch_next_frame")
        return {"codes": self.codes, "eos": self.eos}


class _Request:
    def __init__(self, case, seed):
        rng = np.random.Generator(np.random.Philox(key=[seed, 5]))
        self.prefix, n = case["prefix"], case["prompt"]
        self.engine = _Engine.of(case["weights"], case["kv"], _context_size(self.prefix + n), 2)
        self.ids, self.seed = _synth.random_prompt(n, seed), 1 + seed
        self.voice = _saved_prefix(self.engine, _synth.random_prompt(self.prefix, seed + 1)) if self.prefix else None
        self.kept = _blob(self.engine, self.prefix + n)
        self.slices = []
        clip, first = case["clip"], n // 4
        mask = np.zeros(n, np.uint8)
        mask[first:first + clip] = 1
        codes = rng.integers(0, 4096, size=(CODEBOOKS, clip), dtype=np.int32)
        self.ids[first:first + clip] = SEMANTIC_FIRST + codes[0]
        for lo in range(0, n, SLICE):
            hi = min(n, lo + SLICE)
            a, b = max(lo, first) - first, min(hi, first + clip) - first
            part = None
            if b > a:
                cut = np.ascontiguousarray(codes[:, a:b])
                part = _capi.VqPart(cut.ctypes.data_as(C.POINTER(C.c_int32)), b - a)
                part.keep = cut
            self.slices.append((self.ids[lo:hi], mask[lo:hi], part))
        self.codes, self.eos = (C.c_int32 * CODEBOOKS)(), C.c_int(0)

    def run(self):
        s = _Session(self.engine, 0.8, self.seed)
        if self.prefix:
            s.load(self.voice, self.prefix)
        for ids, mask, part in self.slices:
            s.prefill(ids, mask, part)
        s.save(self.kept, self.prefix + len(self.ids))
        _capi.check(self.engine.lib.s2p_session_next_frame(s.h, self.codes, C.byref(self.eos)), "s2p_session_next_frame")
        s.close()
        return {"codes": np.array(self.codes), "eos": self.eos.value, "cache": self.kept}


class _Layer:
    """Several layers of one shape, called in turn: together with the other states they exceed L2, as a model's do."""
    COPIES = 4

    def __init__(self, case, seed):
        n, k, m = case["n"], case["k"], case["rows"]
        self.lib, self.rows, self.at = _capi.lib(), m, 0
        _capi.check(self.lib.s2p_gemm_init(SLICE), "s2p_gemm_init")
        g = torch.Generator(device="cuda").manual_seed(seed)
        ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        self.keep, self.layers = [], []
        for _ in range(self.COPIES):
            w = (torch.randn(n, k, device="cuda", generator=g) * 0.02).to(torch.bfloat16)
            q = torch.empty(n, k, dtype=torch.int8, device="cuda")
            lin = _capi.Linear(in_features=k, out_features=n, int8_ready=1)
            if case["weights"] == "int4":
                sc = torch.empty(n, k // 32, dtype=torch.float16, device="cuda")
                packed = torch.empty(n, k // 2, dtype=torch.uint8, device="cuda")
                _capi.check(self.lib.s2p_intq_quant(ptr(q), ptr(sc), ptr(w), n, k, 32, 7, 1, None), "s2p_intq_quant")
                _capi.check(self.lib.s2p_int4_pack(ptr(packed), ptr(q), n, k, None), "s2p_int4_pack")
                lin.q_group, lin.q_packed, lin.w_pack.data = 32, 1, packed.data_ptr()
                self.keep += [sc, packed]
            else:
                sc = torch.empty(n, dtype=torch.float32, device="cuda")
                _capi.check(self.lib.s2p_int8_quant(ptr(q), ptr(sc), ptr(w), n, k, None), "s2p_int8_quant")
                lin.w_int8.data = q.data_ptr()
                self.keep += [sc, q]
            lin.w_iscale.data = sc.data_ptr()
            self.layers.append(lin)
            torch.cuda.synchronize()
        self.x = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
        self.y = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")

    def run(self):
        lin = self.layers[self.at % self.COPIES]
        self.at += 1
        _capi.check(self.lib.s2p_linear_forward(C.byref(lin), C.c_void_p(self.x.data_ptr()), C.c_void_p(self.y.data_ptr()), self.rows, _capi.GEMM_INT8,
                                                C.c_void_p(torch.cuda.current_stream().cuda_stream)), "s2p_linear_forward")
        return self.y
