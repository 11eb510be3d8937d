"""The count pass's limit: a long walk gives up where its subtree can be shared
out, and goes on where it cannot (a list would only be walked several times
over).  CPU: the host build of the device runtime."""
import ctypes
import os
import subprocess

import pytest

import test_emu

SO = os.path.join(test_emu.HERE, "emu", "build", "libhvm64_emu_gather.so")
SRC = [os.path.join(test_emu.HERE, "emu", "gather.cpp"), test_emu.SRC[1]]


def _walk(shape, size, limit):
    deps = test_emu.DEPS + SRC
    if not os.path.exists(SO) or any(os.path.getmtime(d) > os.path.getmtime(SO) for d in deps):
        os.makedirs(os.path.dirname(SO), exist_ok=True)
        subprocess.run(["g++", "-std=c++20", "-O2", "-pthread", "-fPIC", "-shared",
                        "-I", os.path.join(test_emu.ROOT, "include"),
                        "-I", os.path.join(test_emu.ROOT, "hvm-64_b200", "csrc"), *SRC, "-o", SO], check=True)
    f = ctypes.CDLL(SO).hvm64emu_limited_walk
    f.argtypes, f.restype = [ctypes.c_int, ctypes.c_uint, ctypes.c_uint], ctypes.c_longlong
    return f(shape, size, limit)


@pytest.mark.parametrize("size", [1, 511, 512, 700, 3000])
def test_a_list_is_walked_to_its_end(size):
    assert _walk(0, size, 1024) == 2 * size + 1


@pytest.mark.parametrize("size", [1, 255, 511])
def test_a_short_tree_is_walked_to_its_end(size):
    assert _walk(1, size, 1024) == 2 * size + 1


@pytest.mark.parametrize("size", [1023, 4000, 100000])
def test_a_long_tree_is_given_up_soon_after_the_limit(size):
    assert -1100 < _walk(1, size, 1024) < -1024
