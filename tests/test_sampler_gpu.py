"""The device sampler against golden sequences of the reference's host sampler and against the CPU oracle."""
import ctypes as C
import os

import numpy as np
import pytest

from _internal_abi import SamplerState

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
GOLD = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
START, EOS = 151678, 151645


class Device:
    def __init__(self, lib, temperature, top_p, penalty, window, seed, rng=(1, 2, 3, 4)):
        s = SamplerState()
        s.temperature, s.top_p, s.rep_penalty, s.window = temperature, top_p, penalty, window
        s.seeded, s.seed31 = 1 if seed else 0, seed & 0x7FFFFFFF
        for i in range(4):
            s.rng[i] = rng[i]
        self.lib, self.state = lib, torch.frombuffer(bytearray(bytes(s)), dtype=torch.uint8).cuda()
        self.at = torch.tensor([self.state.data_ptr()], dtype=torch.int64, device="cuda")
        lib.sample_rows.argtypes = [C.c_void_p, C.c_int64, C.c_void_p, C.c_int64, C.c_void_p, C.c_int] + [C.c_void_p] * 5

    def __call__(self, logits):
        p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        lg = torch.from_numpy(logits.view(np.int16).copy()).cuda()
        tok, sem = torch.zeros(1, dtype=torch.int64, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        codes, eos = torch.zeros(10, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.uint8, device="cuda")
        assert self.lib.sample_rows(p(lg), 4096, C.c_void_p(lg.data_ptr() + 8192), 1, p(self.at), 1, p(tok), p(sem), p(codes), p(eos), None) == 0
        return int(tok), int(sem), int(eos)


def test_golden_sequences(testlib):
    g = np.load(os.path.join(GOLD, "sampler.npz"))
    for tag, temp, seed in (("greedy", 0.0, 0), ("seeded", 0.8, 42), ("seeded_hot", 1.3, 7)):
        d = Device(testlib, temp, 0.8, 1.1, 16, seed)
        for t in range(g["smp_logits"].shape[0]):
            want = tuple(int(g[f"smp_{tag}_{k}"][t]) for k in ("tok", "sem", "eos"))
            assert d(g["smp_logits"][t]) == want, (tag, t)


@pytest.mark.parametrize("temperature,seed", [(0.0, 0), (0.8, 42), (1e-7, 5), (1.5, 77)])
@pytest.mark.parametrize("window", [1, 16, 64])
@pytest.mark.parametrize("spread", [3.0, 0.02])  # the smaller: many equal logits at the thirtieth place and before it
def test_sequences_of_the_oracle(testlib, oracle, temperature, seed, window, spread):
    from oracle import oracle_api as oa
    rng = np.random.default_rng(window)
    sp = C.create_string_buffer(oracle.s2po_sampler_size())
    oracle.s2po_sampler_init(sp, temperature, 0.8, 1.3, window, seed, 0)
    d = Device(testlib, temperature, 0.8, 1.3, window, seed)
    base = rng.standard_normal(4097).astype(np.float32)
    for t in range(70):
        x = (base + 0.3 * rng.standard_normal(4097).astype(np.float32)) * spread
        x[rng.integers(0, 4096, 50)] = -np.inf
        x[rng.integers(0, 4096, 50)] = -0.0
        if t == 20:
            x[4096] = 100.0  # an EOS frame leaves the state alone
        if t == 30:
            x[:] = -np.inf
            x[[5, 6, 4000]] = 1.0
        if t == 40:
            x[:] = 0.0
            x[::2] = -0.0
        lg = oa.f32_to_bf16(x)
        sem, eos = C.c_int32(0), C.c_int32(0)
        tok = oracle.s2po_sample(sp, oa.ptr(lg), int(lg[4096]), 4096, START, EOS, C.byref(sem), C.byref(eos))
        assert d(lg) == (tok, sem.value, eos.value), t


@pytest.mark.parametrize("temperature,seed", [(0.0, 0), (0.8, 42), (0.8, 0)])
@pytest.mark.parametrize("left", [2, 1, 0])
def test_rows_of_nan(testlib, oracle, temperature, seed, left):
    """NaN is never chosen where there is something else; where there is nothing else the frame is EOS, as the oracle's."""
    from oracle import oracle_api as oa
    lg = np.full(4097, 0x7FC0, np.uint16)
    lg[[17, 900][:left]] = [0x3F80, 0x4000][:left]  # 1 and 2
    sp = C.create_string_buffer(oracle.s2po_sampler_size())
    oracle.s2po_sampler_init(sp, temperature, 0.8, 1.1, 16, seed, 0)
    sem, eos = C.c_int32(0), C.c_int32(0)
    tok = oracle.s2po_sample(sp, oa.ptr(lg), int(lg[4096]), 4096, START, EOS, C.byref(sem), C.byref(eos))
    got = Device(testlib, temperature, 0.8, 1.1, 16, seed)(lg)
    if seed == 0 and temperature and left == 2:  # the oracle draws from another stream of random numbers
        assert got[1] in (17, 900) and not got[2]
    else:
        assert got == (tok, sem.value, eos.value) and (got[2] == 0) == (left > 0)
