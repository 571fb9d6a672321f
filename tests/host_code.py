"""Parts of the CUDA sources that hold plain C++ (index arithmetic, scalar arithmetic, host
classes), compiled for the CPU as they stand, between two pieces of their text."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lightspeed_b200", "csrc")

CUDA_WORDS = """
#define __device__
#define __host__
#define __global__
#define __constant__
#define __forceinline__ inline
#define __restrict__
"""


def source_part(name, begin, end):
    text = open(os.path.join(CSRC, name)).read()
    assert text.count(begin) == 1, "%s: %r" % (name, begin)
    start = text.index(begin)
    return text[start:text.index(end, start + len(begin))]


def compile_host(tmp_path, code):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    src, lib = str(tmp_path / "part.cpp"), str(tmp_path / "part.so")
    with open(src, "w") as fh:
        fh.write(code)
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-Wno-unknown-pragmas", "-shared", "-fPIC", "-I", CSRC,
                    src, "-o", lib], check=True)
    return ctypes.CDLL(lib)
