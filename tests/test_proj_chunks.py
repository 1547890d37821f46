"""The projection kernels' chunk tables after a failed allocation, on the CPU
(tests/cpp/proj_chunks_check.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "proj_chunks_check.cpp")


def test_a_failed_build_is_built_again(tmp_path):
    exe = os.path.join(str(tmp_path), "proj_chunks_check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", SRC, "-I/usr/local/cuda/include",
                        "-I" + os.path.join(ROOT, "include"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "bad=0", r.stdout + r.stderr
