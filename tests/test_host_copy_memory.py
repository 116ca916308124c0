"""The staged host copies (csrc/host_copy.cu, plain C++ over the CUDA runtime)
against a runtime that copies in place, with every host allocation made while a
copier is built refused in turn: no call may end the process, and what can be
copied arrives whole."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "csharp_linearalgebra_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_refused_allocations(tmp_path):
    exe = tmp_path / "harness"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(CUDA, "include"), "-I" + CSRC, "-x", "c++",
                    os.path.join(HERE, "host_copy_harness.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stderr)
