"""Kernels that start before the one in front of them has ended: what they read behind their wait has to be read there.

A load through a `const __restrict__` parameter, or `__ldg`, may be moved in front of the wait, and whether the compiler does so shows in no
output until it happens.  So the sources are held to the rule of launch.cuh: a parameter that is read is not restricted, or it comes out of the wait
itself, and behind the wait, or in a helper that may be called there, nothing uses `__ldg`."""
import glob
import os
import re

import pytest

CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "s2pro-native_b200", "csrc", "cuda")


def closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise ValueError("unbalanced " + pair)


def kernels(text):
    """(name, parameter list, span of the body) of every kernel defined in the text."""
    for m in re.finditer(r"\bk_\w+\(", text):
        head = text.rfind("__global__", 0, m.start())
        if head < 0 or re.search(r"[;{}]", text[head:m.start()]):
            continue
        end = closing(text, m.end() - 1, "()")
        body = text.index("{", end)
        if text[end + 1:body].strip():
            continue
        yield m.group()[:-1], text[m.end():end], (body, closing(text, body, "{}"))


def broken_rules(text, header=False):
    found, spans = [], []
    for name, params, (lo, hi) in kernels(text):
        body = text[lo:hi]
        wait = re.search(r"\bgrid_wait(_for)?\(", body)
        spans.append((lo, lo + wait.start() if wait else hi))
        if not wait:
            continue
        through = {a.strip() for args in re.findall(r"\bgrid_wait_for\(([^)]*)\)", body) for a in args.split(",")}
        for p in params.split(","):
            if re.search(r"\bconst\b[^,]*\*\s*__restrict__", p) and p.split()[-1] not in through:
                found.append(f"{name}: {p.split()[-1]} is read as constant, but does not come out of the wait")
    if header or re.search(r"\bgrid_wait(_for)?\(", text):
        found += ["__ldg behind a wait, or in a helper: " + text[m.start():m.start() + 60].split("\n")[0]
                  for m in re.finditer(r"\b__ldg\(", text) if not any(lo < m.start() < hi for lo, hi in spans)]
    return found


@pytest.mark.parametrize("path", sorted(p for p in glob.glob(os.path.join(CUDA, "*.cu*")) if not p.endswith("launch.cuh")), ids=os.path.basename)
def test_kernels_read_behind_their_wait(path):
    with open(path) as f:
        text = re.sub(r"/\*.*?\*/|//[^\n]*", "", f.read(), flags=re.S)
    assert not broken_rules(text, path.endswith(".cuh"))


def test_the_rule_sees_what_it_is_for():
    kernel = "__global__ void __launch_bounds__(32) k_a(float* y, const float* __restrict__ x) { int i = 0; %s y[i] = %s; }"
    assert not broken_rules(kernel % ("grid_wait_for(x);", "x[i]"))
    assert not broken_rules((kernel % ("grid_wait();", "x[i]")).replace("__restrict__ ", ""))
    assert not broken_rules(kernel % ("", "__ldg(x)"))
    assert len(broken_rules(kernel % ("grid_wait();", "x[i]"))) == 1
    assert len(broken_rules(kernel % ("grid_wait_for(x);", "__ldg(x)"))) == 1
    helper = "__device__ float of(const float* p) { return __ldg(p); } "
    assert len(broken_rules(helper + kernel % ("grid_wait_for(x);", "of(x)"))) == 1
    assert len(broken_rules(helper, header=True)) == 1
