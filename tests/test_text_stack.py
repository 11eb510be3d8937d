"""Short normal forms are formatted on the calling thread, which may have a
small stack: lists that nest a few hundred levels deep, and trees, on a thread
with 64 KiB.  Each runs in a process of its own, which an overflow would end.
CPU."""
import os
import subprocess
import sys

import pytest

import test_emu

SO = os.path.join(test_emu.HERE, "emu", "build", "libhvm64_texts.so")
SRC = [os.path.join(test_emu.HERE, "emu", "texts.cpp"), test_emu.SRC[1]]
RUN = """
import ctypes, sys
f = ctypes.CDLL(sys.argv[1]).hvm64emu_text
f.argtypes = [ctypes.c_int, ctypes.c_uint, ctypes.c_size_t, ctypes.c_char_p, ctypes.c_size_t]
f.restype = ctypes.c_size_t
buf = ctypes.create_string_buffer(1 << 16)
n = f(int(sys.argv[2]), int(sys.argv[3]), 64 << 10, buf, 1 << 16)
assert n == len(buf.value)
print(buf.value.decode())
"""


def _tree(k, size):
    return f"({_tree(2 * k, size)} {_tree(2 * k + 1, size)})" if k <= size else "0"


@pytest.mark.parametrize("shape,size", [(0, n) for n in (1, 62, 63, 64, 65, 400, 511, 512)] + [(1, 1), (1, 300), (1, 511)])
def test_texts_on_a_small_stack(shape, size):
    deps = [os.path.join(test_emu.ROOT, "hvm-64_b200", "csrc", "host.hpp"), *SRC]
    if not os.path.exists(SO) or any(os.path.getmtime(d) > os.path.getmtime(SO) for d in deps):
        os.makedirs(os.path.dirname(SO), exist_ok=True)
        subprocess.run(["g++", "-std=c++20", "-O2", "-pthread", "-fPIC", "-shared",
                        "-I", os.path.join(test_emu.ROOT, "include"),
                        "-I", os.path.join(test_emu.ROOT, "hvm-64_b200", "csrc"), *SRC, "-o", SO], check=True)
    r = subprocess.run([sys.executable, "-c", RUN, SO, str(shape), str(size)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    want = _tree(1, size) if shape else "(0 " * size + "0" + ")" * size
    assert r.stdout.strip() == want
