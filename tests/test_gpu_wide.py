"""The wide part kernel on the GPU against the oracle: every gate kind it holds
at the smallest state it takes, odd sizes and every tile size, after a slot
permutation, and with frames carried from call to call; complex128 <= 1e-12,
complex64 <= 1e-5."""
import numpy as np
import pytest

from hisvsim_b200 import abi, circuits, partition
from hisvsim_b200.gates import Gate, part_offsets, to_records
from test_k1_wide import _mixed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(abi.C128, 1e-12), (abi.C64, 1e-5)])
@pytest.mark.parametrize("hint", [0, 10, 11, 12])
@pytest.mark.parametrize("n", [10, 11, 12, 13, 16, 17])
def test_wide_passes_match_oracle(port, n, hint, dtype, tol):
    gates = _mixed(n, 3, n) + circuits.random_u3_cz(n, 3, n)
    want = port.run(n, to_records(gates))
    parts = partition.partition_frontier(gates, 8, free_diagonal=True)
    rec, offs = part_offsets(partition.parts_to_gates(gates, parts))
    rng = np.random.default_rng(n)
    prev = abi.set_tile_qubits(hint)
    try:
        st = abi.State(n, dtype)
        st.run_parts(rec, offs)
        assert np.abs(st.amplitudes() - want).max() <= tol
        st.set_basis(0)
        fr = abi.Frames(n)
        for p in range(len(offs) - 1):
            st.run_part_carry(fr, rec[offs[p]:offs[p + 1]])
            if p % 3 == 1:  # the factors follow their qubits
                st.permute_bits([int(v) for v in rng.permutation(n)[:4]])
        st.flush(fr)
        assert np.abs(st.amplitudes() - want).max() <= tol
    finally:
        abi.set_tile_qubits(prev)


@pytest.mark.parametrize("dtype,tol", [(abi.C128, 1e-12), (abi.C64, 1e-5)])
@pytest.mark.parametrize("m", [(1, 2e-17, 0, 1), (1, 0, 2e-17, 1), (1, 2e-13, 0, 1j), (0, 1, 1, 2e-17)])
def test_gates_diagonal_to_rounding(port, m, dtype, tol):
    """Custom gates with a rounding residue off (or on) the diagonal, among gates that flip."""
    n = 12
    near = Gate("C1", (2,), params=m)
    gates = ([Gate("H", (q,)) for q in range(n)] + [Gate("X", (0,)), Gate("RY", (1,), params=(3.0,)), near]
             + circuits.random_layered(n, 3, 5) + [near])
    want = port.run(n, to_records(gates))
    rec, offs = part_offsets([gates[:n + 3], gates[n + 3:n + 40], gates[n + 40:]])
    st = abi.State(n, dtype)
    st.run_parts(rec, offs)
    assert np.abs(st.amplitudes() - want).max() <= tol
    st.set_basis(0)
    fr = abi.Frames(n)
    for p in range(len(offs) - 1):
        st.run_part_carry(fr, rec[offs[p]:offs[p + 1]])
    st.flush(fr)
    assert np.abs(st.amplitudes() - want).max() <= tol


@pytest.mark.parametrize("odd", [None, Gate("H", (0,), (1,)), Gate("RXX", (3, 1), params=(0.3,))])
def test_timed_parts_match_the_plain_call(port, odd):
    """run_parts_timed: the bits of run_parts in complex64, also where one part holds a
    gate outside the wide form; its amplitudes in complex128."""
    n = 12
    parts = [[Gate("H", (q,)) for q in range(n)] + [Gate("RY", (q,), params=(3.0,)) for q in range(n)],
             ([odd] if odd else []) + [Gate("U3", (2,), params=(2.5, 0.3, 1.0))], _mixed(n, 2, 6)]
    rec, offs = part_offsets(parts)
    want = port.run(n, rec)
    for dtype, tol in ((abi.C64, 1e-5), (abi.C128, 1e-12)):
        a, b = abi.State(n, dtype), abi.State(n, dtype)
        a.run_parts(rec, offs)
        ms = b.run_parts_timed(rec, offs)
        assert len(ms) == len(parts)
        x, y = a.amplitudes(), b.amplitudes()
        assert dtype != abi.C64 or np.array_equal(x, y)
        assert max(np.abs(x - want).max(), np.abs(y - want).max()) <= tol


@pytest.fixture(scope="module")
def many_tiles(port):
    """A circuit on 24 qubits: four tiles per CTA and more at every tile size."""
    n = 24
    gates = circuits.random_u3_cz(n, 1, n) + [Gate("X", (0,), (n - 1,)), Gate("SWAP", (1, n - 2))]
    rec, offs = part_offsets(partition.parts_to_gates(gates, partition.partition_frontier(gates, 10)))
    return n, rec, offs, port.run(n, to_records(gates))


@pytest.mark.parametrize("dtype,tol", [(abi.C128, 1e-12), (abi.C64, 1e-5)])
@pytest.mark.parametrize("hint", [0, 10, 11, 12])
def test_many_tiles_per_cta(many_tiles, dtype, tol, hint):
    """Tiles drawn from the state's counter: it is back at 0 after every pass (a second
    run gives the same bits), two states at once on two streams have their own, and a
    captured run replays."""
    import torch

    n, rec, offs, want = many_tiles
    prev = abi.set_tile_qubits(hint)
    try:
        st = [abi.State(n, dtype) for _ in range(2)]
        st[0].run_parts(rec, offs)
        first = st[0].amplitudes()
        assert np.abs(first - want).max() <= tol
        streams = [torch.cuda.Stream() for _ in range(2)]
        for s, x in zip(st, streams):
            s.set_basis(0, stream=x.cuda_stream)
        for _ in range(2):
            for s, x in zip(st, streams):
                s.set_basis(0, stream=x.cuda_stream)
                s.run_parts(rec, offs, stream=x.cuda_stream)
        torch.cuda.synchronize()
        assert all(np.array_equal(s.amplitudes(), first) for s in st)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(streams[0]):
            g.capture_begin(capture_error_mode="thread_local")
            st[0].set_basis(0, stream=streams[0].cuda_stream)
            st[0].run_parts(rec, offs, stream=streams[0].cuda_stream)
            g.capture_end()
        for _ in range(3):
            st[0].load(np.zeros(1 << n, st[0].np_dtype))
            g.replay()
            torch.cuda.synchronize()
            assert np.array_equal(st[0].amplitudes(), first)
    finally:
        abi.set_tile_qubits(prev)


def test_passes_without_low_slots_are_not_slower_than_the_general_form():
    """29 qubits, complex128, passes whose 12 targets leave no low slot (runs of 16
    bytes): the wide form is the one taken, so the general form (8 amplitudes per
    thread) does not run the same pass faster."""
    n = 29
    st = abi.State(n)
    for qs in ([3, 5, 7, 12, 13, 14, 15, 16, 17, 24, 27, 28], [7, 12, 13, 14, 15, 17, 18, 19, 20, 23, 26, 28]):
        rec, offs = part_offsets([[Gate("U3", (q,), params=(0.3 + q, 0.1, 0.2)) for q in qs for _ in range(2)]])
        ms = {}
        for r in (3, 4):
            prev = abi.set_k1_reg_bits(r)
            try:
                ms[r] = min(float(st.run_parts_timed(rec, offs)[0]) for _ in range(4))
            finally:
                abi.set_k1_reg_bits(prev)
        assert ms[4] <= ms[3], ms
