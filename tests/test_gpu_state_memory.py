"""Device memory of small states is kept when they are destroyed: a new state
starts from |0..0> whatever its memory held, work still in flight on another
stream does not reach it, threads do not share blocks, and what is kept stays
bounded."""
import threading

import numpy as np
import pytest

from hisvsim_b200 import abi, circuits
from hisvsim_b200.gates import to_records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dtype", [(1, abi.C64), (10, abi.C128), (20, abi.C128), (21, abi.C128)])
def test_new_state_starts_fresh(n, dtype):
    import torch

    rec = to_records(circuits.random_u3_cz(n, 3, n)) if n > 1 else None
    side = torch.cuda.Stream()
    for _ in range(4):
        st = abi.State(n, dtype)
        a = st.raw()
        assert a[0] == 1 and not a[1:].any()
        if rec is not None:
            for _ in range(5):  # left in flight on a stream of the caller's
                st.run_part(rec, stream=side.cuda_stream)
        st.close()


def test_threads_do_not_share_blocks(port):
    n = 12
    rec = [to_records(circuits.random_layered(n, 4, s)) for s in range(4)]
    want = [port.run(n, r) for r in rec]
    bad = []

    def work(k):
        abi.set_device(0)
        for _ in range(20):
            st = abi.State(n)
            st.run_part(rec[k])
            if np.abs(st.amplitudes() - want[k]).max() > 1e-12:
                bad.append(k)
            st.close()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad


def test_kept_memory_is_bounded():
    import torch

    torch.cuda.init()
    abi.State(4).close()
    before = torch.cuda.mem_get_info()[0]
    for n in list(range(1, 23)) * 2:
        states = [abi.State(n) for _ in range(3)]
        [s.close() for s in states]
    # 32 MiB of states and the granularity of their mappings
    assert before - torch.cuda.mem_get_info()[0] <= 96 << 20


def test_states_come_and_go_beside_a_capture():
    """A thread makes, uses and destroys states while another captures a stream
    (thread-local mode, as hs_batch does): the capture stays valid."""
    import torch

    x = torch.zeros(1024, device="cuda")
    side = torch.cuda.Stream()
    rec = to_records(circuits.random_layered(10, 2, 1))
    abi.State(10).close()
    err = []

    def states():
        try:
            abi.set_device(0)
            for n in (4, 10, 12):
                for stream in (None, side.cuda_stream):
                    st = abi.State(n)
                    if n == 10:
                        st.run_part(rec, stream=stream)
                    st.close()
        except Exception as e:  # noqa: BLE001
            err.append(e)

    g = torch.cuda.CUDAGraph()
    cap = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(cap):
        g.capture_begin(capture_error_mode="thread_local")
        x.add_(1.0)
        t = threading.Thread(target=states)
        t.start()
        t.join()
        x.add_(1.0)
        g.capture_end()
    g.replay()
    torch.cuda.synchronize()
    assert not err
    assert bool((x == 2.0).all())


def test_kept_memory_of_many_states_is_bounded():
    """Eight states of 16 MiB destroyed together leave 32 MiB and the granularity
    of their mappings."""
    import torch

    torch.cuda.init()
    abi.State(4).close()
    before = torch.cuda.mem_get_info()[0]
    for n in (20, 19, 20):
        states = [abi.State(n) for _ in range(8)]
        [s.close() for s in states]
    assert before - torch.cuda.mem_get_info()[0] <= 48 << 20


_RESET = """
import ctypes, glob, os, sys
import numpy as np, torch
from hisvsim_b200 import abi
rt = ctypes.CDLL(glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib", "libcudart.so.*"))[0])
for n in (4, 12, 20):
    st = abi.State(n)
    st.norm2()
    st.close()
assert rt.cudaDeviceReset() == 0
try:  # states need the library's kernels in the new context; its memory must be new either way
    for n in (4, 12, 20):
        st = abi.State(n)
        a = st.raw()
        assert a[0] == 1 and not a[1:].any()
        assert abs(st.norm2() - 1) < 1e-12
        st.close()
    print("usable")
except abi.HisvError as e:
    print("refused", e)
"""


def test_reset_device_leaves_no_stale_blocks():
    """After a device reset no block of the old context is handed out."""
    import subprocess
    import sys

    r = subprocess.run([sys.executable, "-c", _RESET], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.startswith(("usable", "refused"))
    assert "illegal" not in r.stdout
