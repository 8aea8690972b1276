"""The host part of hs_measure (place_samples): every sample in the chunk its point
falls into, in work items of a bounded number of samples, so that many samples of
a small state (one chunk) are searched by many blocks."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("measure") / "libplace.so")
    csrc = os.path.join(ROOT, "hisvsim_b200", "csrc")
    cmd = ["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I/usr/local/cuda/include",
           "-I" + os.path.join(ROOT, "include"), "-I" + csrc, os.path.join(csrc, "measure.cpp"),
           os.path.join(ROOT, "tests", "emu", "measure_probe.cpp"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        pytest.fail("build failed:\n" + r.stderr[-3000:])
    return ctypes.CDLL(out)


@pytest.mark.parametrize("chunks,n", [(1, 1), (1, 127), (1, 129), (1, 100000), (8, 3000), (64, 10), (3, 0)])
def test_work_items(lib, chunks, n):
    rng = np.random.default_rng(chunks * 7 + n)
    mass = rng.uniform(size=chunks)
    if chunks > 3:
        mass[2] = 0.0
    mass *= 0.95 / mass.sum()  # some points lie beyond the mass
    u = np.sort(rng.uniform(size=n))
    most = int(lib.samples_per_block())
    assert 1 <= most <= 1024
    items = np.zeros((n + 1, 3), np.uint64)
    bases = np.zeros(n + 1)
    placed = ctypes.c_uint32(99)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    k = lib.place(p(mass), chunks, 16, p(u), n, most, p(items), p(bases), ctypes.byref(placed))
    cum = np.concatenate([[0.0], np.cumsum(mass)])
    where = np.searchsorted(cum[1:], u, side="right")  # chunk of each point
    assert placed.value == int((where < chunks).sum())
    nxt = 0
    for i in range(k):
        first, s0, ns = (int(v) for v in items[i])
        assert s0 == nxt and 1 <= ns <= most
        c = first >> 16
        assert np.all(where[s0:s0 + ns] == c) and bases[i] == cum[c]
        nxt += ns
    assert nxt == placed.value
    assert k <= chunks + n // most
