"""The redex queue's first tickets over 2^28 + 2^20 runs of one ring (two days
of 0.6 ms calls): each above every word earlier runs left in the ring, so that
the ring reads as empty.  CPU."""
import ctypes
import os
import subprocess

import test_emu

SO = os.path.join(test_emu.HERE, "emu", "build", "libhvm64_emu_tickets.so")
SRC = [os.path.join(test_emu.HERE, "emu", "tickets.cpp"), test_emu.SRC[1]]


def test_every_run_starts_above_the_words_of_earlier_ones():
    deps = test_emu.DEPS + SRC
    if not os.path.exists(SO) or any(os.path.getmtime(d) > os.path.getmtime(SO) for d in deps):
        os.makedirs(os.path.dirname(SO), exist_ok=True)
        subprocess.run(["g++", "-std=c++20", "-O2", "-pthread", "-fPIC", "-shared",
                        "-I", os.path.join(test_emu.ROOT, "include"),
                        "-I", os.path.join(test_emu.ROOT, "hvm-64_b200", "csrc"), *SRC, "-o", SO], check=True)
    f = ctypes.CDLL(SO).hvm64emu_tickets
    f.argtypes, f.restype = [ctypes.c_ulonglong], ctypes.c_ulonglong
    assert f((1 << 28) + (1 << 20)) == 0
