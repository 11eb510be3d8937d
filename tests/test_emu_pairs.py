"""Reclaiming the nodes an interaction consumes when other lanes take the other
ends of its wires meanwhile: whatever CASes lose, and however many, every node
is reclaimed once.  CPU: the host build of the device runtime."""
import ctypes
import os
import subprocess

import pytest

import test_emu

SO = os.path.join(test_emu.HERE, "emu", "build", "libhvm64_emu_pairs.so")
SRC = [os.path.join(test_emu.HERE, "emu", "pairs.cpp"), test_emu.SRC[1]]


def _lib():
    deps = test_emu.DEPS + SRC
    if not os.path.exists(SO) or any(os.path.getmtime(d) > os.path.getmtime(SO) for d in deps):
        os.makedirs(os.path.dirname(SO), exist_ok=True)
        subprocess.run(["g++", "-std=c++20", "-O2", "-pthread", "-fPIC", "-shared", "-DHVM_EMU_CHECK_ALLOC",
                        "-I", os.path.join(test_emu.ROOT, "include"),
                        "-I", os.path.join(test_emu.ROOT, "hvm-64_b200", "csrc"), *SRC, "-o", SO], check=True)
    L = ctypes.CDLL(SO)
    L.hvm64emu_pairs.argtypes = [ctypes.c_uint, ctypes.c_int, ctypes.c_int]
    L.hvm64emu_pairs.restype = ctypes.c_ulonglong
    return L


@pytest.mark.parametrize("chase", [0, 1])
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("nodes", [1, 2, 3, 4])
def test_every_consumed_node_is_reclaimed_once(nodes, order, chase):
    assert _lib().hvm64emu_pairs(nodes, order, chase) == 0
