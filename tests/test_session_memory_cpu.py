"""Device memory of sessions when the GPU runs out of it: the host sources with a small stand-in for the CUDA runtime (no GPU)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "s2pro-native_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def run(tmp_path, name, sources):
    exe = str(tmp_path / name)
    # what these tests do not reach stays unresolved
    subprocess.run(["gcc", "-std=c11", "-D_GNU_SOURCE", "-O1", "-g", "-I", os.path.join(CSRC, "host"), "-I", os.path.join(CSRC, "..", "..", "include"),
                    "-I", os.path.join(CUDA, "include"), os.path.join(HERE, "host", name + ".c")] + [os.path.join(CSRC, "host", s) for s in sources] +
                   ["-o", exe, "-lm", "-lpthread", "-no-pie", "-Wl,--unresolved-symbols=ignore-all"], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, f"{name}.c:{out.returncode} failed\n{out.stderr}"


def test_sessions_and_pools(tmp_path):
    run(tmp_path, "session_memory", ["session.c", "core.c"])
