"""Kept device memory, the host logic (kept_blocks.h): bounded, the oldest given
up for new sizes, nothing handed out of a context that is gone, and given back
when an allocation fails."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("kept") / "libkept.so")
    cmd = ["g++", "-O1", "-std=c++17", "-fPIC", "-shared",
           "-I" + os.path.join(ROOT, "hisvsim_b200", "csrc"),
           os.path.join(ROOT, "tests", "emu", "kept_blocks_probe.cpp"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        pytest.fail("build failed:\n" + r.stderr[-3000:])
    L = ctypes.CDLL(out)
    u64, sz, P, lg = ctypes.c_uint64, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_long
    L.pool_new.restype = P
    L.pool_take.argtypes, L.pool_take.restype = [P, u64, sz], lg
    L.pool_put.argtypes = [P, u64, lg, sz, P]
    L.pool_drain.argtypes = [P, u64, P]
    L.alloc_tries.argtypes = [P, ctypes.c_int, P]
    return L


class Pool:  # of 1000 bytes
    def __init__(self, lib):
        self.lib, self.q, self.buf = lib, lib.pool_new(), (ctypes.c_long * 64)()

    def take(self, ctx, size):
        return self.lib.pool_take(self.q, ctx, size)

    def put(self, ctx, p, size):
        return list(self.buf[:self.lib.pool_put(self.q, ctx, p, size, self.buf)])

    def drain(self, ctx):
        return list(self.buf[:self.lib.pool_drain(self.q, ctx, self.buf)])


def test_new_sizes_replace_the_oldest(lib):
    q = Pool(lib)
    assert q.put(1, 11, 500) == [] and q.put(1, 12, 500) == []
    assert q.put(1, 13, 100) == [11]  # two large blocks do not shut a size out
    assert q.take(1, 100) == 13 and q.take(1, 100) == 0
    assert q.put(1, 14, 600) == [12]
    assert q.put(1, 15, 1001) == [15]  # never more than the bound
    assert q.put(1, 16, 1000) == [14]
    assert q.drain(1) == [16] and q.drain(1) == [] and q.take(1, 1000) == 0


def test_blocks_of_a_lost_context_are_not_handed_out(lib):
    q = Pool(lib)
    q.put(3, 31, 400)
    assert q.take(4, 400) == 0 and q.drain(4) == []  # neither reused nor freed
    assert q.put(4, 41, 700) == []  # (31 is forgotten with its context)
    assert q.put(3, 32, 100) == [32]
    assert q.take(4, 400) == 0 and q.take(4, 700) == 41
    assert q.put(0, 5, 100) == [5] and q.take(0, 100) == 0  # context unknown


@pytest.mark.parametrize("errors,kept,want,tries", [((0, 9), 1, 0, 1), ((2, 0), 1, 0, 2),
                                                    ((2, 2), 1, 2, 2), ((2, 0), 0, 2, 1), ((7, 0), 1, 7, 1)])
def test_allocation_gives_kept_memory_back(lib, errors, kept, want, tries):
    n = ctypes.c_int()
    assert lib.alloc_tries((ctypes.c_int * 2)(*errors), kept, ctypes.byref(n)) == want
    assert n.value == tries
