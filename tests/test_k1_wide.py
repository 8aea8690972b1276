"""Wide K1 programs on the CPU: the library's planner (plan.cpp) compiled with
the host emulator tests/emu/k1_wide_emu.cpp, which runs the planned programs as
the kernel does and range-checks every offset.  Compared with the oracle
(port.c) over every form of chunk that takes the wide path: each gate kind it
holds with its bits in registers, threads and outer slots, slot orders, both
data types, tile sizes from 2^10 to 2^12, carried and flushed frames.
Tolerances: 1e-12 (complex128) as for every plain form, 1e-5 (complex64)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from hisvsim_b200 import circuits, partition
from hisvsim_b200.gates import Gate, part_offsets, to_records

CSRC = os.path.join(ROOT, "hisvsim_b200", "csrc")
SRCS = [os.path.join(ROOT, "tests", "emu", "k1_wide_emu.cpp"), os.path.join(CSRC, "plan.cpp"),
        os.path.join(CSRC, "gatemath.cpp")]


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("wide") / "libwideemu.so")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I/usr/local/cuda/include",
           "-I" + os.path.join(ROOT, "include"), "-I" + CSRC] + SRCS + ["-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        pytest.fail("emulator build failed:\n" + r.stderr[-3000:])
    lib = ctypes.CDLL(out)
    P = ctypes.c_void_p
    lib.wide_parts_run.argtypes = [ctypes.c_int, ctypes.c_int, P, P, ctypes.c_int, P, ctypes.c_int,
                                   ctypes.c_int, P, P]
    lib.wide_last_error.restype = ctypes.c_char_p
    lib.wide_plan_time.argtypes = [ctypes.c_int, ctypes.c_int, P, P, ctypes.c_int, P, P]

    def run(n, parts, dtype=0, hint=0, mode=0, q2s=None):
        """Amplitudes in qubit order of the parts run from |0...0>, and the statistics."""
        rec, offs = part_offsets(parts)
        q2s = np.arange(n, dtype=np.int32) if q2s is None else np.asarray(q2s, dtype=np.int32)
        a = np.zeros(1 << n, complex)
        a[0] = 1
        st = np.zeros(5, np.int32)
        rc = lib.wide_parts_run(n, dtype, rec.ctypes.data, offs.ctypes.data, len(offs) - 1,
                                q2s.ctypes.data, hint, mode, a.ctypes.data, st.ctypes.data)
        if rc:
            raise RuntimeError(lib.wide_last_error().decode())
        x = np.arange(1 << n)
        slot = sum(((x >> q) & 1) << int(q2s[q]) for q in range(n))
        return a[slot], dict(zip(["passes", "wide", "groups", "steps", "tables"], st.tolist()))
    run.lib = lib
    return run


def _mixed(n, layers, seed):
    """Every gate kind of the wide form on random qubits."""
    rng = np.random.default_rng(seed)
    u = lambda: float(rng.uniform(0, 2 * np.pi))  # noqa: E731
    g = []
    for _ in range(layers):
        for q in range(n):
            g.append(Gate("U3", (q,), params=(u(), u(), u())) if rng.integers(2) else Gate("H", (q,)))
        for _ in range(n):
            q = [int(v) for v in rng.permutation(n)[:4]]
            k = int(rng.integers(11))
            g.append([Gate("X", (q[0],), (q[1],)), Gate("X", (q[0],), (q[1], q[2])),
                      Gate("Z", (q[0],), (q[1],)), Gate("Z", (q[0],), (q[1], q[2])),
                      Gate("SWAP", (q[0], q[1])), Gate("RZZ", (q[0], q[1]), params=(u(),)),
                      Gate("U1", (q[0],), (q[1],), params=(u(),)),
                      Gate("C1", (q[0],), (q[1], q[2]), params=(1.0, 0.0, 0.0, np.exp(1j * u()))),
                      Gate("T", (q[0],)), Gate("RZ", (q[0],), params=(u(),)),
                      Gate("RZZ", (q[0], q[1]), (q[2],), params=(u(),))][k])
    return g


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("hint", [0, 10, 11, 12])
@pytest.mark.parametrize("kind,n,k", [("mixed", 10, 10), ("mixed", 13, 8), ("u3cz", 14, 9),
                                      ("layered", 13, 7), ("qft", 12, 6), ("qft", 13, 10)])
def test_wide_programs_match_oracle(emu, port, kind, n, k, hint, dtype):
    gates = {"mixed": lambda: _mixed(n, 4, 7), "u3cz": lambda: circuits.random_u3_cz(n, 8, 3),
             "layered": lambda: circuits.random_layered(n, 8, 4),
             "qft": lambda: circuits.qft(n, 2)[0]}[kind]()
    want = port.run(n, to_records(gates))
    tol = 1e-5 if dtype else 1e-12
    for split in (partition.partition_acyclic, partition.partition_dfs):
        parts = partition.parts_to_gates(gates, split(gates, k))
        for mode in (0, 1, 2):
            got, st = emu(n, parts, dtype=dtype, hint=hint, mode=mode)
            assert st["wide"] == st["passes"] > 0
            # (the flush of the pending factors may take a pass of its own)
            assert mode != 2 or st["passes"] <= len(parts) + 1
            assert np.abs(got - want).max() <= tol


@pytest.mark.parametrize("seed", range(6))
def test_any_slot_order(emu, port, seed):
    """The chunk's qubits in shuffled slots (after a redistribution)."""
    n = 13
    gates = _mixed(n, 3, 100 + seed)
    want = port.run(n, to_records(gates))
    q2s = np.random.default_rng(seed).permutation(n)
    parts = partition.parts_to_gates(gates, partition.partition_frontier(gates, 8, free_diagonal=True))
    for dtype, tol in ((0, 1e-12), (1, 1e-5)):
        for mode in (0, 2):
            got, st = emu(n, parts, dtype=dtype, mode=mode, q2s=q2s)
            assert st["wide"] == st["passes"]
            assert np.abs(got - want).max() <= tol


def test_program_limits(emu, port):
    """Parts at the limits of one program: many rotations of one qubit in a row
    (a step each), more conditional phases and sign flips than a program holds,
    and a flush with every qubit pending."""
    rng = np.random.default_rng(3)
    n = 12
    u = lambda: tuple(float(v) for v in rng.uniform(0, 2 * np.pi, 3))  # noqa: E731
    deep = [g for i in range(150) for g in (Gate("U3", (3,), params=u()), Gate("Z", (3,), (i % 3,)))]
    many = [Gate("U3", (q,), params=u()) for q in range(n)]
    for i in range(300):
        a, b = (int(x) for x in rng.choice(n, 2, replace=False))
        many.append(Gate("U1", (a,), (b,), params=(u()[0],)) if i % 2 else Gate("Z", (a,), (b,)))
    many += [Gate("U3", (q,), params=u()) for q in range(n)]
    swaps = [g for i in range(140) for g in (Gate("SWAP", tuple(int(x) for x in rng.choice(n, 2, replace=False))),
                                             Gate("RY", (i % n,), params=(3.0,)))]
    # phases and pairs on bits that flips keep turning over
    turned = [g for i in range(120) for g in (
        Gate("RY", (i % 5,), params=(3.0,)), Gate("Z", (i % 5,), ((i + 1) % 5,)),
        Gate("C1", (i % 5,), ((i + 1) % 5, (i + 2) % 5), params=(1.0, 0.0, 0.0, 1j)),
        Gate("U1", (i % 5,), (5 + i % 7,), params=(0.1 + i,)))]
    for gates in (deep, many, swaps, turned):
        want = port.run(n, to_records(gates))
        for mode in (0, 1, 2):
            got, st = emu(n, [gates], mode=mode)
            assert st["wide"] == st["passes"] > 0
            assert np.abs(got - want).max() <= 1e-12


def test_passes_take_gates_of_later_parts(emu, port):
    """Parts bounded by every touched qubit leave room in the tile: one call takes
    fewer passes than parts, also when the gates in between stay behind."""
    n = 16
    for gates in (circuits.random_layered(n, 6, 9), circuits.random_u3_cz(n, 6, 9), _mixed(n, 3, 5)):
        want = port.run(n, to_records(gates))
        parts = partition.parts_to_gates(gates, partition.partition_acyclic(gates, 6))
        got, st = emu(n, parts, mode=2)
        assert st["passes"] < len(parts)
        assert np.abs(got - want).max() <= 1e-12
        # complex64 calls keep a pass per part
        assert emu(n, parts, dtype=1, mode=2)[1]["passes"] >= len(parts)


def test_flips_and_custom_gates(emu, port):
    """Rotations beyond the pivot (X and Y among them) next to every gate that
    meets a flipped bit, and frames that custom gates leave far from 1 between
    calls: those calls do without flips."""
    rng = np.random.default_rng(17)
    n = 12
    g = []
    for _ in range(5):
        for q in range(n):
            g.append([Gate("X", (q,)), Gate("Y", (q,)), Gate("RY", (q,), params=(3.0,)),
                      Gate("U3", (q,), params=(2.9, float(rng.uniform(0, 6)), 1.0))][int(rng.integers(4))])
        for _ in range(8):
            q = [int(v) for v in rng.permutation(n)[:4]]
            g.append([Gate("Z", (q[0],), (q[1],)), Gate("Z", (q[0],), (q[1], q[2])),
                      Gate("X", (q[0],), (q[1], q[2])), Gate("SWAP", (q[0], q[1])),
                      Gate("RZZ", (q[0], q[1]), params=(0.7,)),
                      Gate("C1", (q[0],), (q[1], q[2], q[3]), params=(1.0, 0.0, 0.0, 1j))][int(rng.integers(6))])
    want = port.run(n, to_records(g))
    for split, k in ((partition.partition_acyclic, 12), (partition.partition_dfs, 6)):
        parts = partition.parts_to_gates(g, split(g, k))
        for mode in (0, 1, 2):
            got, st = emu(n, parts, mode=mode)
            assert st["wide"] == st["passes"]
            assert np.abs(got - want).max() <= 1e-12
            got, _ = emu(n, parts, dtype=1, mode=mode)
            assert np.abs(got - want).max() <= 1e-5
    # a first call whose custom diagonal leaves a factor of 1e4 pending
    parts = [[Gate("H", (q,)) for q in range(n)] + [Gate("C1", (3,), params=(1.0, 0.0, 0.0, 1e4))], g]
    want = port.run(n, to_records([x for p in parts for x in p]))
    got, _ = emu(n, parts, mode=0)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


def test_other_gates_keep_the_general_form(emu):
    """Gates outside the wide form (dense controlled, two-qubit dense, custom
    non-unitary diagonals, controlled swaps) and small states are not taken."""
    wide = [Gate("H", (q,)) for q in range(11)]
    for g in (Gate("H", (0,), (1,)), Gate("RXX", (0, 1), params=(0.3,)),
              Gate("C1", (0,), (1,), params=(0.5, 0.0, 0.0, 1.0)), Gate("SWAP", (0, 1), (2,))):
        _, st = emu(11, [wide + [g]])
        assert st["passes"] == 1 and st["wide"] == 0
    _, st = emu(9, [[Gate("H", (q,)) for q in range(9)]])
    assert st["passes"] == 1 and st["wide"] == 0


def test_gates_diagonal_to_rounding_are_not_refused(emu):
    """A custom gate with one off-diagonal entry of exactly 0 and the other a
    rounding residue, next to gates that flip: applied as a matrix where it is no
    rotation (lower left 0), and its call does without flips."""
    n = 12
    base = [Gate("H", (q,)) for q in range(n)] + [Gate("X", (0,)), Gate("RY", (1,), params=(3.0,))]
    for m, wide in (((1, 2e-17, 0, 1), False), ((1, 0, 2e-17, 1), True),
                    ((1, 2e-13, 0, 1j), False), ((5e-324, 1, 1, 0), True), ((0, 1, 1, 2e-17), True)):
        gate = Gate("C1", (2,), params=m)
        for parts in ([base + [gate]], [[gate] + base], [base, [gate], base]):
            for dtype in (0, 1):
                for mode in (0, 1, 2):
                    _, st = emu(n, parts, dtype=dtype, mode=mode)
                    assert (st["wide"] == st["passes"]) == wide


@pytest.mark.parametrize("dtype", [0, 1])
def test_long_calls_are_planned_as_they_run(emu, dtype):
    """A call of many gates hands its first pass over early and plans in linear
    time: the first of 80 000 gates' passes within a fifth of the whole (best of
    three), eight times the gates within sixteen times the time."""
    n = 20
    def plan(count):
        gates = circuits.random_layered(n, count // n, 3)[:count]
        rec = to_records(gates)
        offs = np.append(np.arange(0, count, 25), count).astype(np.int32)
        best = (1e9, 1e9, 0)
        for _ in range(3):
            passes, sec = ctypes.c_int32(), (ctypes.c_double * 2)()
            assert emu.lib.wide_plan_time(n, dtype, rec.ctypes.data, offs.ctypes.data, len(offs) - 1,
                                          ctypes.byref(passes), sec) == 0
            best = min(best, (sec[1], sec[0], passes.value))
        return best
    short, _, few = plan(10000)
    total, first, many = plan(80000)
    assert first <= total / 5
    assert total <= 16 * short
    assert many <= 9 * few


def test_timed_calls_plan_as_plain_ones(emu, port):
    """hs_parts_run_timed's passes (mode 3): in complex64 those of hs_parts_run, a part
    outside the wide form among them (the emulator leaves such passes out in both);
    in complex128 the same amplitudes to rounding."""
    n = 11
    for odd in ([], [Gate("H", (0,), (1,))], [Gate("RXX", (0, 1), params=(0.3,))]):
        parts = [[Gate("H", (q,)) for q in range(n)] + [Gate("RY", (q,), params=(3.0,)) for q in range(n)],
                 odd + [Gate("U3", (2,), params=(2.5, 0.3, 1.0))], _mixed(n, 1, 6)]
        plain, a = emu(n, parts, dtype=1, mode=2)
        timed, b = emu(n, parts, dtype=1, mode=3)
        assert a == b and np.array_equal(plain, timed)
        if not odd:
            want = port.run(n, to_records([g for p in parts for g in p]))
            assert np.abs(emu(n, parts, mode=3)[0] - want).max() <= 1e-12


@pytest.mark.parametrize("dtype,tol", [(0, 1e-12), (1, 1e-4)])
def test_calls_of_several_windows(emu, port, dtype, tol):
    """More gates than one planning window holds: parts that end at, before and beyond
    its border, one longer than a window, empty ones, frames carried across."""
    n = 11
    gates = circuits.random_layered(n, 150, 8) + _mixed(n, 6, 9)
    want = port.run(n, to_records(gates))
    for sizes in ([25], [1024], [1023, 1, 2], [7, 0, 1100, 30], [len(gates)]):
        parts, i = [], 0
        while i < len(gates):
            k = sizes[len(parts) % len(sizes)]
            parts.append(gates[i:i + k])
            i += k
        got, st = emu(n, parts, dtype=dtype, mode=2)
        assert st["wide"] == st["passes"]
        assert np.abs(got - want).max() <= tol
        if dtype == 1:
            timed, _ = emu(n, parts, dtype=dtype, mode=3)
            assert np.array_equal(got, timed)


def test_windows_grow_with_the_state(emu):
    """A call of 1960 gates on 33 qubits is one window (fewer passes than its halves
    planned apart)."""
    def passes(n, parts):
        rec, offs = part_offsets(parts)
        k, sec = ctypes.c_int32(), (ctypes.c_double * 2)()
        assert emu.lib.wide_plan_time(n, 0, rec.ctypes.data, offs.ctypes.data, len(offs) - 1,
                                      ctypes.byref(k), sec) == 0
        return k.value
    gates = circuits.random_u3_cz(33, 40, 1)
    parts = partition.parts_to_gates(gates, partition.partition_frontier(gates, 9))
    cut = next(i for i in range(len(parts)) if sum(map(len, parts[:i + 1])) > 1024)
    assert passes(33, parts) < passes(33, parts[:cut]) + passes(33, parts[cut:])
