"""A communicator's work from several threads, on the caller's default stream and
on the library's own: cpp/test_stream.cpp with the CUDA runtime replaced by a
model, so no GPU is needed."""
import os
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_work_of_several_threads_is_ordered(tmp_path):
    exe = tmp_path / "test_stream"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + str(ROOT / "include"),
                    "-I" + str(ROOT / "spmv_b200" / "csrc"), "-I" + CUDA + "/include",
                    str(ROOT / "tests" / "cpp" / "test_stream.cpp"),
                    str(ROOT / "spmv_b200" / "csrc" / "stream.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
