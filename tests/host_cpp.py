"""Builds and runs a small host C++ program against the library's headers, with stand-ins for the CUDA
calls they make: the decisions of host code that no GPU run can be asked to get wrong."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fesom2_gb300", "csrc")


def cuda_include() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


def run(tmp_path, source: str, timeout: float = 60.0) -> str:
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(source)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, "-I", cuda_include(), str(src), "-o", str(exe), "-lpthread"],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=timeout)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
