"""Programs that run the library's device code on the CPU (cuda_runtime.h here
stands in for CUDA's), for tests of single device functions and of kernels
whose faults a GPU must not meet."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))


def compile_program(source, tmp_path, sanitize=False):
    """Compiles C++ `source` (it includes "argent_b200/csrc/...") and returns
    the program's path."""
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    src, exe = os.path.join(tmp_path, "program.cpp"), os.path.join(tmp_path, "program")
    with open(src, "w") as f:
        f.write(source)
    flags = ["-fsanitize=address,undefined", "-fno-sanitize-recover=undefined", "-g"] if sanitize else []
    p = subprocess.run([cxx, "-std=c++20", "-O1", "-ffp-contract=off", "-pthread", *flags, "-I", HERE, "-I", ROOT, src,
                        "-o", exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[:3000]
    return exe


def run(exe, data=b"", args=(), timeout=300):
    """Runs a program on `data` (its standard input) and returns its output."""
    p = subprocess.run([exe, *args], input=data, stdout=subprocess.PIPE, stderr=subprocess.PIPE, timeout=timeout)
    assert p.returncode == 0, p.stderr.decode(errors="replace")[-3000:]
    return p.stdout
