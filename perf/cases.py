"""The work whose time counts: the simulator's public calls over the range of
sizes, circuits, data types and forms that its tests, its benchmark and its
QASM front end use.

A case is a dict of plain values; ``kind`` says which entry points it takes:

* ``parts``   -- a circuit from a basis state in one ``State.run_parts`` call
  (what ``qasm.simulate`` and the benchmark do);
* ``loop``    -- the same through the pybind module, one
  ``gather_and_execute_on`` per part, amplitudes read back (a program written
  for the reference's Python API);
* ``gates``   -- one ``State.apply`` per gate on a state in hand
  (``BoundGate::apply``);
* ``fused``   -- the precision form, ``State.run_fused`` on complex64;
* ``batch``   -- the batching form, ``QaoaBatch.run`` with new angles;
* ``swap``    -- the qubit redistribution, ``State.permute_bits``;
* ``readout`` -- norm, marginals, <ZZ> of a ring and samples of one state;
* ``train``   -- the learned form: one training call of the cost model, then
  the pricing of every part.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from hisvsim_b200 import abi, partition
from hisvsim_b200 import svsimulator_py_wrapper as svsim
from hisvsim_b200.gates import Gate, part_offsets, to_records

FEATURES = 43  # inputs of the cost model (abi.num_part_features())
HIDDEN = 64


def listed():
    return [
        # a small program through the reference's Python API: launches, host
        # planning and allocation are all there is
        {"name": "loop layered 13q", "kind": "loop", "circuit": "layered", "n": 13, "layers": 6,
         "split": "acyclic", "limit": 7},
        # the parity workload: every common gate, a state that fits the L2
        {"name": "parts layered 20q", "kind": "parts", "circuit": "layered", "n": 20, "layers": 20,
         "split": "acyclic", "limit": 10, "dtype": "c128"},
        # parts as the reference bounds them (every touched qubit), an odd count
        {"name": "parts u3cz 27q", "kind": "parts", "circuit": "u3cz", "n": 27, "layers": 8,
         "split": "frontier", "limit": 9, "dtype": "c128"},
        # the benchmark's circuit and parts (non-diagonal targets bounded),
        # at a size whose passes stream HBM
        {"name": "parts u3cz 30q", "kind": "parts", "circuit": "u3cz", "n": 30, "layers": 8,
         "split": "free", "limit": 9, "dtype": "c128"},
        # the QFT: mostly controlled phases, then swaps
        {"name": "parts qft 29q", "kind": "parts", "circuit": "qft", "n": 29, "layers": 1,
         "split": "free", "limit": 7, "dtype": "c128"},
        # the plain form in single precision, as the learned form runs it
        {"name": "parts u3cz 30q c64", "kind": "parts", "circuit": "u3cz", "n": 30, "layers": 8,
         "split": "frontier", "limit": 10, "dtype": "c64"},
        # gate by gate, every gate a sweep
        {"name": "gates layered 26q", "kind": "gates", "circuit": "layered", "n": 26, "count": 24,
         "dtype": "c128"},
        # the precision form on the benchmark's circuit
        {"name": "fused u3cz 29q", "kind": "fused", "circuit": "u3cz", "n": 29, "layers": 8,
         "split": "frontier", "limit": 6},
        # a parameter sweep over instances of mixed sizes
        {"name": "batch 48 of 14-23q", "kind": "batch", "count": 48, "low": 14, "high": 23, "p": 4},
        # three low slots exchanged with three high ones
        {"name": "swap 29q", "kind": "swap", "n": 29, "pairs": 3, "dtype": "c128"},
        # what is read from a state at the end of a run
        {"name": "readout 28q", "kind": "readout", "n": 28, "probs": 4, "shots": 512,
         "dtype": "c128"},
        # the cost model: an epoch in minibatches, then inference
        {"name": "train 8192", "kind": "train", "rows": 8192, "epochs": 1, "batch": 256},
    ]


def draw(rng):
    kind = rng.choice(["parts", "parts", "parts", "parts", "loop", "gates", "fused", "batch",
                       "swap", "readout", "train"])
    if kind in ("parts", "loop"):
        circuit = rng.choice(["layered", "u3cz", "qft", "qaoa"])
        n = rng.randint(12, 29) if kind == "parts" else rng.randint(8, 18)
        split = rng.choice(["acyclic", "frontier", "free", "dfs"])
        c = {"kind": kind, "circuit": circuit, "n": n, "split": split,
             "layers": 1 if circuit in ("qft", "qaoa") else rng.randint(3, 9 if n > 24 else 20),
             "limit": rng.randint(6, 10)}
        if kind == "parts":
            c["dtype"] = rng.choice(["c128", "c128", "c64"])
        return c
    if kind == "gates":
        return {"kind": "gates", "circuit": "layered", "n": rng.randint(10, 28),
                "count": rng.randint(8, 32), "dtype": rng.choice(["c128", "c64"])}
    if kind == "fused":
        return {"kind": "fused", "circuit": rng.choice(["u3cz", "layered"]),
                "n": rng.randint(14, 29), "layers": rng.randint(3, 8),
                "split": rng.choice(["frontier", "dfs", "acyclic"]), "limit": 6}
    if kind == "batch":
        low = rng.randint(8, 18)
        return {"kind": "batch", "count": rng.randint(4, 48), "low": low,
                "high": rng.randint(low, 22), "p": rng.randint(1, 6)}
    if kind == "swap":
        return {"kind": "swap", "n": rng.randint(16, 29), "pairs": rng.randint(1, 7),
                "dtype": rng.choice(["c128", "c64"])}
    if kind == "readout":
        return {"kind": "readout", "n": rng.randint(12, 28), "probs": rng.randint(1, 8),
                "shots": int(2 ** rng.uniform(4, 10)), "dtype": rng.choice(["c128", "c64"])}
    return {"kind": "train", "rows": int(2 ** rng.uniform(7, 14)), "epochs": rng.randint(1, 2),
            "batch": rng.choice([64, 128, 256])}


# ---- circuits as plain tuples (name, targets, controls, parameters) ------------


def _matching(rng, n):
    perm = rng.permutation(n)
    return [(int(perm[2 * i]), int(perm[2 * i + 1])) for i in range(n // 2)]


def _graph(rng, n):
    """A 3-regular simple graph (one vertex of degree 2 when n is odd)."""
    while True:
        deg = np.full(n, 3)
        if n % 2:
            deg[int(rng.integers(n))] = 2
        stubs = rng.permutation(np.repeat(np.arange(n), deg)).reshape(-1, 2)
        edges = {(int(min(a, b)), int(max(a, b))) for a, b in stubs if a != b}
        if len(edges) == len(stubs):
            return sorted(edges)


def _circuit(case, seed):
    """(gates, index of the initial basis state)."""
    rng = np.random.default_rng(seed)
    n, name, out, x = case["n"], case["circuit"], [], 0
    if name == "qft":
        x = int(rng.integers(0, 1 << n))
        for i in range(n - 1, -1, -1):
            out.append(("H", (i,), (), ()))
            for j in range(i - 1, -1, -1):
                phi = 2.0 * math.pi / (1 << (i - j + 1))
                out.append(("C1", (i,), (j,), (1.0, 0.0, 0.0, complex(math.cos(phi), math.sin(phi)))))
        out += [("SWAP", (i, n - 1 - i), (), ()) for i in range(n // 2)]
    elif name == "qaoa":
        edges = _graph(rng, n)
        out += [("H", (q,), (), ()) for q in range(n)]
        for _ in range(2):
            g, b = float(rng.uniform(0, math.pi)), float(rng.uniform(0, math.pi))
            out += [("RZZ", e, (), (g,)) for e in edges]
            out += [("RX", (q,), (), (b,)) for q in range(n)]
    else:
        for _ in range(case.get("layers", 4)):
            for q in range(n):
                g = "U3" if name == "u3cz" else ["H", "X", "S", "T", "RZ", "U3"][int(rng.integers(6))]
                params = {"RZ": 1, "U3": 3}.get(g, 0)
                out.append((g, (q,), (), tuple(float(v) for v in rng.uniform(0, 2 * math.pi, params))))
            for a, b in _matching(rng, n):
                flip = name != "u3cz" and rng.integers(2) == 0
                out.append(("X" if flip else "Z", (b,), (a,), ()))
    return out, x


def _gate(g):
    return Gate(g[0], g[1], g[2], g[3])


def _parts(case, gates):
    k = min(case["limit"], case["n"])
    split = case["split"]
    if split == "acyclic":
        parts = partition.partition_acyclic(gates, k)
    elif split == "dfs":
        parts = partition.partition_dfs(gates, k)
    else:
        parts = partition.partition_frontier(gates, k, free_diagonal=split == "free")
    return partition.parts_to_gates(gates, parts)


def _bound(g):
    """A gate as the reference's Python API writes it."""
    if g.name in ("U3",):
        ag = svsim.AggregateGate_3(g.name, *g.params)
    elif g.name == "C1":
        ag = svsim.AggregateGate_C1(g.name, *g.params)
    elif g.params:
        ag = svsim.AggregateGate_1(g.name, *g.params)
    else:
        ag = svsim.AggregateGate_0(g.name)
    return svsim.BoundGate(svsim.AggregateGateFactory(ag), list(g.controls), list(g.targets))


# ---- states ---------------------------------------------------------------------


class _DeviceArray:
    """The amplitudes of a State, described for torch (no copy)."""

    def __init__(self, st):
        p = abi._vp()
        abi.check(abi.lib().hs_state_device_ptr(st.h, abi.ctypes.byref(p)))
        self.owner = st
        self.__cuda_array_interface__ = {
            "shape": (1 << st.n, 2), "typestr": "<f8" if st.dtype == abi.C128 else "<f4",
            "data": (p.value, False), "version": 2}


def _state(n, dtype):
    """A state and its slot-ordered amplitudes as a (2^n, 2) tensor."""
    st = abi.State(n, abi.C128 if dtype == "c128" else abi.C64)
    return st, torch.as_tensor(_DeviceArray(st), device="cuda")


def _random_amps(n, dtype, seed):
    """Amplitudes of a deep circuit's state: normal, normalised."""
    real = torch.float64 if dtype == "c128" else torch.float32
    gen = torch.Generator("cuda").manual_seed(seed)
    a = torch.randn((1 << n, 2), dtype=real, device="cuda", generator=gen)
    return a.mul_(2.0 ** (-0.5 * (n + 1)))


def _swap_pairs(case, seed):
    """Disjoint (low slot, high slot) pairs."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    np_ = min(case["pairs"], n // 2)
    low = rng.choice(n // 2, np_, replace=False)
    high = n // 2 + rng.choice(n - n // 2, np_, replace=False)
    return [int(v) for ab in zip(low, high) for v in ab]


def _ring(n):
    return [(q, (q + 1) % n) for q in range(n)]


def _instances(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["count"]):
        n = case["low"] + i % (case["high"] - case["low"] + 1)
        out.append((n, _graph(rng, n), rng.uniform(0, math.pi, case["p"]),
                    rng.uniform(0, math.pi / 2, case["p"])))
    return out


def _rows(case, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, 1, (case["rows"], FEATURES)).astype(np.float32)
    y = (np.sin(x[:, :8].sum(axis=1)) + x[:, 8:16].sum(axis=1) * 0.25).astype(np.float32)
    p = np.concatenate([v for k in (FEATURES, HIDDEN, HIDDEN)
                        for v in (rng.uniform(-1, 1, HIDDEN * k) * math.sqrt(6.0 / k),
                                  np.zeros(HIDDEN))] +
                       [rng.uniform(-1, 1, HIDDEN) * math.sqrt(6.0 / HIDDEN), np.zeros(1)])
    return x, y, p.astype(np.float32)


# ---- the calls ------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("parts", "loop", "fused"):
        tuples, s["x"] = _circuit(case, seed)
        parts = _parts(case, [_gate(g) for g in tuples])
        if kind == "loop":
            s["parts"] = [[_bound(g) for g in p] for p in parts]
            # the reference's StateVector starts from |0..0>
            s["prep"] = [_bound(Gate("X", (q,))) for q in range(case["n"]) if (s["x"] >> q) & 1]
        else:
            s["rec"], s["offs"] = part_offsets(parts)
            s["st"], s["amp"] = _state(case["n"], "c64" if kind == "fused" else case["dtype"])
    elif kind == "gates":
        tuples, _ = _circuit(case, seed)
        s["recs"] = [to_records([_gate(g)]) for g in tuples[-case["count"]:]]
        s["st"], s["amp"] = _state(case["n"], case["dtype"])
        s["amp"].copy_(_random_amps(case["n"], case["dtype"], seed))
    elif kind == "swap":
        s["pairs"] = _swap_pairs(case, seed)
        s["st"], s["amp"] = _state(case["n"], case["dtype"])
        s["amp"].copy_(_random_amps(case["n"], case["dtype"], seed))
    elif kind == "readout":
        s["st"], s["amp"] = _state(case["n"], case["dtype"])
        s["amp"].copy_(_random_amps(case["n"], case["dtype"], seed))
        s["qubits"] = [int(q) for q in
                       np.random.default_rng(seed).integers(0, case["n"], case["probs"])]
        s["seed"] = seed
    elif kind == "batch":
        inst = _instances(case, seed)
        s["gammas"] = np.array([i[2] for i in inst])
        s["betas"] = np.array([i[3] for i in inst])
        s["batch"] = abi.QaoaBatch(inst, case["p"])
    else:
        s["xs"], s["ys"], s["p0"] = _rows(case, seed)
        s["mlp"] = abi.Mlp(FEATURES, 0)
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "parts":
        s["st"].set_basis(s["x"])
        s["st"].run_parts(s["rec"], s["offs"])
        return s["amp"]
    if kind == "fused":
        s["st"].set_basis(s["x"])
        s["st"].run_fused(s["rec"], s["offs"], 0)
        return s["amp"]
    if kind == "loop":
        sv = svsim.StateVector(case["n"], 1)
        if s["prep"]:
            svsim.gather_and_execute_on(sv, s["prep"])
        for part in s["parts"]:
            svsim.gather_and_execute_on(sv, part)
        return sv.amplitudes()
    if kind == "gates":
        for rec in s["recs"]:
            s["st"].apply(rec)
        return s["amp"]
    if kind == "swap":
        s["st"].permute_bits(s["pairs"])
        return s["amp"]
    if kind == "readout":
        st = s["st"]
        return {"norm": st.norm2(), "prob": np.array([st.probability(q) for q in s["qubits"]]),
                "zz": st.expect_zz(_ring(case["n"])),
                "shots": st.measure(list(range(case["n"])), case["shots"], s["seed"])}
    if kind == "batch":
        s["batch"].set_params(s["gammas"], s["betas"])
        expect, _ = s["batch"].run()
        # the angles' result per instance, and the smallest instance's state
        return {"expect": expect, "state": s["batch"].state(0)}
    mlp = s["mlp"]
    mlp.set_params(s["p0"])
    losses = mlp.train(s["xs"], s["ys"], case["epochs"], case["batch"], 1e-3, 5)
    return {"loss": losses, "params": mlp.params(), "price": mlp.predict(s["xs"])}


# ---- what a pass cannot do without -------------------------------------------------

# flops per amplitude: a one-qubit rotation by real shears takes 7 multiply-adds
# per amplitude pair; a diagonal factor one complex product on the amplitudes
# its qubits select
_ROTATION, _FACTOR = 7.0, 6.0


def _gate_flops(g):
    name, nt, nc = g[0], len(g[1]), len(g[2])
    if name in ("SWAP", "I") or (name in ("X", "Z") and nc):
        return 0.0
    if name in ("S", "T", "RZ", "Z"):
        return 0.0  # a factor that later rotations of the qubit take in
    if name == "RZZ":
        return _FACTOR
    if name == "C1":
        return _FACTOR / 2 ** (nt + nc)
    return _ROTATION / 2 ** nc


def work(case):
    kind = case["kind"]
    if kind in ("parts", "loop", "fused", "gates"):
        tuples, _ = _circuit(case, 0)
        amp = 8 if kind == "fused" or case.get("dtype") == "c64" else 16
        if kind == "gates":  # every call reads and writes the state
            tuples = tuples[-case["count"]:]
            moved = 2 * amp * len(tuples)
        else:
            moved = amp
        return {"bytes": float(moved << case["n"]),
                "flops": sum(_gate_flops(g) for g in tuples) * float(1 << case["n"])}
    if kind == "swap":
        amp = 8 if case["dtype"] == "c64" else 16
        return {"bytes": 2.0 * amp * (1 << case["n"]) * (1 - 0.5 ** case["pairs"]), "flops": 0.0}
    if kind == "readout":
        amp = 8 if case["dtype"] == "c64" else 16
        # the calls that the API has: the norm, each marginal, one for the
        # ring, one for the samples; a marginal needs half the state
        reads = 1 + 0.5 * case["probs"] + 1 + 1
        return {"bytes": reads * amp * (1 << case["n"]),
                "flops": (3.0 * (3 + case["probs"]) + case["n"]) * (1 << case["n"])}
    if kind == "batch":
        amps = sum(1 << (case["low"] + i % (case["high"] - case["low"] + 1))
                   for i in range(case["count"]))
        return {"bytes": 8.0 * amps, "flops": 0.0 + amps * case["p"] * case["low"] * 4.0}
    weights = HIDDEN * (FEATURES + 2 * HIDDEN + 1)
    return {"bytes": 4.0 * case["rows"] * (FEATURES + 2),
            "flops": 2.0 * weights * case["rows"] * (3 * case["epochs"] + 1)}


# ---- the same in 64 bits ------------------------------------------------------------


def _matrix(name, p):
    r = math.sqrt(0.5)
    e = lambda a: complex(math.cos(a), math.sin(a))  # noqa: E731
    if name == "H":
        return (r, r, r, -r)
    if name == "X":
        return (0.0, 1.0, 1.0, 0.0)
    if name == "RX":
        return (math.cos(p[0] / 2), -1j * math.sin(p[0] / 2), -1j * math.sin(p[0] / 2),
                math.cos(p[0] / 2))
    if name == "U3":
        t, f, l = p
        c, s = math.cos(t / 2), math.sin(t / 2)
        return (c * e(-(f + l) / 2), -s * e((l - f) / 2), s * e((f - l) / 2), c * e((f + l) / 2))
    if name == "C1":
        return p
    if name == "RZ":
        return (e(-p[0] / 2), 0.0, 0.0, e(p[0] / 2))
    return {"Z": (1.0, 0.0, 0.0, -1.0), "S": (1.0, 0.0, 0.0, 1j), "T": (1.0, 0.0, 0.0, e(math.pi / 4))}[name]


def _sub(psi, n, bits):
    """The amplitudes whose index bits are as given, as a view."""
    shape, index, prev = [], [], n
    for q in sorted(bits, reverse=True):
        shape += [1 << (prev - 1 - q), 2]
        index += [slice(None), bits[q]]
        prev = q
    return psi.view(shape + [1 << prev])[tuple(index)]


def _apply(psi, n, g):
    name, ts, cs, p = g
    on = {q: 1 for q in cs}
    if name == "SWAP":
        a, b = _sub(psi, n, {ts[0]: 1, ts[1]: 0}), _sub(psi, n, {ts[0]: 0, ts[1]: 1})
        t = a.clone()
        a.copy_(b)
        b.copy_(t)
        return
    if name == "RZZ":
        for i in range(4):
            a = (-1 if i in (0, 3) else 1) * p[0] / 2
            _sub(psi, n, {ts[0]: i & 1, ts[1]: i >> 1}).mul_(complex(math.cos(a), math.sin(a)))
        return
    m = _matrix(name, p)
    a, b = _sub(psi, n, {**on, ts[0]: 0}), _sub(psi, n, {**on, ts[0]: 1})
    if m[1] == 0 and m[2] == 0:
        for v, f in ((a, m[0]), (b, m[3])):
            if f != 1:
                v.mul_(f)
        return
    t = a.clone()
    a.mul_(m[0]).add_(b, alpha=m[1])
    b.mul_(m[3]).add_(t, alpha=m[2])


def _simulate(n, tuples, x):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[x] = 1.0
    for g in tuples:
        _apply(psi, n, g)
    return psi


def _exact_batch(case, seed):
    expect, state = [], None
    for i, (n, edges, gammas, betas) in enumerate(_instances(case, seed)):
        idx = torch.arange(1 << n, device="cuda")
        cut = torch.zeros(1 << n, dtype=torch.float64, device="cuda")
        for a, b in edges:
            cut += ((idx >> a) ^ (idx >> b)) & 1
        psi = torch.full((1 << n,), 2.0 ** (-0.5 * n), dtype=torch.complex128, device="cuda")
        for g, b in zip(gammas, betas):
            psi *= torch.exp(0.5j * float(g) * (2.0 * cut - len(edges)))
            for q in range(n):
                _apply(psi, n, ("RX", (q,), (), (2.0 * float(b),)))
        expect.append(float((torch.view_as_real(psi).square().sum(1) * cut).sum()))
        state = psi if i == 0 else state
    return {"expect": np.array(expect), "state": state.cpu().numpy()}


def _shuffles(seed, rows, epochs):
    """The training call's row orders (splitmix64, Fisher-Yates)."""
    mask, state = (1 << 64) - 1, seed
    for _ in range(epochs):
        perm = list(range(rows))
        for i in range(rows - 1, 0, -1):
            state = (state + 0x9E3779B97F4A7C15) & mask
            z = ((state ^ (state >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        yield np.array(perm)


def _unpack(p):
    out, at = [], 0
    for rows, k in ((HIDDEN, FEATURES), (HIDDEN, HIDDEN), (HIDDEN, HIDDEN), (1, HIDDEN)):
        out += [p[at:at + rows * k].reshape(rows, k), p[at + rows * k:at + rows * k + rows]]
        at += rows * (k + 1)
    return out


def _exact_train(case, seed):
    x, y, p = (v.astype(np.float64) for v in _rows(case, seed))
    m, v, step, losses = np.zeros_like(p), np.zeros_like(p), 0, []
    # the learning rate and the decay rates are single precision arguments
    lr, b1, b2, eps = (float(np.float32(f)) for f in (1e-3, 0.9, 0.999, 1e-8))

    def forward(x):
        w = _unpack(p)
        hs = [x]
        for k in range(3):
            hs.append(np.maximum(hs[-1] @ w[2 * k].T + w[2 * k + 1], 0.0))
        return w, hs, (hs[-1] @ w[6].T + w[7])[:, 0]

    for perm in _shuffles(5, len(x), case["epochs"]):
        total = 0.0
        for at in range(0, len(x), case["batch"]):
            rows = perm[at:at + case["batch"]]
            w, hs, f = forward(x[rows])
            r = f - y[rows]
            total += float((r * r).sum())
            d = (2.0 / len(rows) * r)[:, None]
            grads = []
            for k in (3, 2, 1, 0):
                grads = [(d.T @ hs[k]).reshape(-1), d.sum(axis=0)] + grads
                d = (d @ w[2 * k]) * (hs[k] > 0)
            g = np.concatenate(grads)
            step += 1
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            p = p - lr * (m / (1 - b1 ** step)) / (np.sqrt(v / (1 - b2 ** step)) + eps)
        losses.append(total / len(x))
    return {"loss": np.array(losses), "params": p, "price": forward(x)[2]}


def exact(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind in ("parts", "fused", "loop"):
        tuples, x = _circuit(case, seed)
        psi = _simulate(n, tuples, x)
        return psi.cpu().numpy() if kind == "loop" else torch.view_as_real(psi)
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    amps = _random_amps(n, case["dtype"], seed).double()
    if kind == "gates":
        psi = torch.view_as_complex(amps)
        for g in _circuit(case, seed)[0][-case["count"]:]:
            _apply(psi, n, g)
        return amps
    if kind == "swap":
        pairs = _swap_pairs(case, seed)
        for a, b in zip(pairs[0::2], pairs[1::2]):
            _apply(torch.view_as_complex(amps), n, ("SWAP", (a, b), (), ()))
        return amps
    mass = amps.square_().sum(1)
    zz = [float(sum((1 - 2 * (i ^ j)) * _sub(mass, n, {a: i, b: j}).sum()
                    for i in (0, 1) for j in (0, 1))) for a, b in _ring(n)]
    rng = np.random.default_rng(seed)
    return {"norm": float(mass.sum()),
            "prob": np.array([float(_sub(mass, n, {int(q): 0}).sum())
                              for q in rng.integers(0, n, case["probs"])]),
            "zz": np.array(zz), "shots": None}
