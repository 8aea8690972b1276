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
