"""The rank order of the nonlocal scatter's records, on the CPU (tests/cpp/rank_tables_check.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "rank_tables_check.cpp")
LIBDIR = os.path.join(ROOT, "inq-wannier-fork_b200", "lib")


def test_rank_order(pb, tmp_path):
    exe = os.path.join(str(tmp_path), "rank_tables_check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", SRC, "-I/usr/local/cuda/include", "-L" + LIBDIR, "-linqb200",
                        "-L/usr/local/cuda/lib64", "-lcudart", "-Wl,-rpath," + LIBDIR, "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.count("bad=0") == 4, r.stdout + r.stderr
