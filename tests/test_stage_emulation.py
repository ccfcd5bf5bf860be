"""CPU check of the staged passes (no GPU): tests/stage_emu/stage_emu.cpp runs
gate lists through the library's own planner and the kernel's own per-thread
functions.  The state must match the oracle to the rounding of its precision,
every amplitude must be loaded and stored exactly once per pass, every
shared-memory slot written and read exactly once per stage change, and passes
without renamed qubits must be free of bank conflicts.
"""
import ctypes as C
import os
import subprocess
import time

import numpy as np
import pytest

from oracle.pyoracle import OracleState
from qpanda_b200 import circuits
from qpanda_b200.capi import OP, lib
from tests.golden.make_golden import every_gate_circuit

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIBDIR = os.path.join(ROOT, "qpanda_b200", "_lib")
C64, C128 = 0, 1
# FP32: a few roundings of 6e-8 per gate on amplitudes below 1, ~150 gates
TOL = {C64: 1e-6, C128: 1e-14}


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    lib()                                     # the library must be built
    out = str(tmp_path_factory.mktemp("stage_emu") / "libstage_emu.so")
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(ROOT, "tests", "stage_emu", "stage_emu.cpp"),
           "-I" + os.path.join(ROOT, "qpanda_b200", "csrc"), "-I" + os.path.join(ROOT, "include"), "-L" + LIBDIR,
           "-lqsb200", "-Wl,-rpath=" + LIBDIR, "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    E = C.CDLL(out)
    E.stage_emu_error.restype = C.c_char_p
    return E


def plan(E, n, gates, dtype, state=None):
    """Run (or with state=None only plan) the list; (passes, stages, conflicts, ops, small)."""
    g = np.ascontiguousarray(gates)
    st = (C.c_longlong * 5)()
    r = E.stage_emu_apply(None if state is None else state.ctypes.data_as(C.c_void_p), n,
                          g.ctypes.data_as(C.c_void_p), len(g), dtype, st)
    assert r == 0, E.stage_emu_error().decode()
    return list(st)


def phases_and_swaps(n, seed):
    """Ladders on shared hubs, repeated and multi-controlled phases, swaps and
    controlled gates whose controls and targets lie anywhere."""
    rng = np.random.default_rng(seed)
    spec = []
    for _ in range(60):
        a, b, c = (int(x) for x in rng.permutation(n)[:3])
        spec += [("CR", (a, b), 0.3), ("CR", (a, c), -0.7), ("CR", (b, a), 1.1), ("H", (c,)), ("SWAP", (b, c)),
                 ("RZ", (a,), 0.4), ("CNOT", (c, a)), ("RX", (b,), 2.5), ("RY", (b,), 2.9), ("X", (c,))]
    g = circuits.make_gates(spec)
    for k in range(0, len(g), 7):             # QRunes CONTROL lists on every kind of gate
        free = [q for q in range(n) if q not in g["q"][k][:2]]
        g["nctrl"][k] = 2
        g["ctrl"][k][:2] = rng.permutation(free)[:2]
    return g


LISTS = {
    "layers": lambda n: circuits.random_layers(n, 5, n, iswap_frac=0.3),
    "qft": circuits.qft,
    "every": lambda n: every_gate_circuit(n, 11 + n),
    "ansatz": lambda n: circuits.vqe_ansatz(n, 3, n),
    "phases": lambda n: phases_and_swaps(n, n),
    "long": lambda n: circuits.random_layers(n, 40, n),         # several parameter blocks' worth
}


@pytest.mark.parametrize("dtype", [C64, C128])
@pytest.mark.parametrize("n", [8, 9, 10, 12, 13, 15])
@pytest.mark.parametrize("kind", list(LISTS))
def test_passes_match_oracle(emu, kind, n, dtype):
    rng = np.random.default_rng(7 * n + dtype)
    init = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    init /= np.linalg.norm(init)
    gates = LISTS[kind](n)
    st = init.copy()
    passes, stages, conflicts, ops, small = plan(emu, n, gates, dtype, st)
    o = OracleState(n)
    o.set_state(init)
    o.apply(gates)
    assert np.abs(st - o.state()).max() < TOL[dtype] * (4 if kind == "long" else 1)
    if n >= 12 and kind in ("layers", "ansatz"):
        assert conflicts == 0


def swaps(n, kind):
    """Lists that end in swaps of disjoint qubits: the reversal of all, of all
    but the lowest four, random pairs (some qubits left alone)."""
    if kind == "all":
        pairs = [(k, n - 1 - k) for k in range(n // 2)]
    elif kind == "upper":
        pairs = [(4 + k, n - 1 - k) for k in range((n - 4) // 2)]
    else:
        q = np.random.default_rng(n).permutation(n)
        pairs = [(int(q[2 * k]), int(q[2 * k + 1])) for k in range(n // 2 - 1)]
    return circuits.make_gates([("RY", (q,), 0.3 + q) for q in range(0, n, 3)] + [("SWAP", p) for p in pairs])


@pytest.mark.parametrize("dtype", [C64, C128])
@pytest.mark.parametrize("n", [13, 16, 17, 18])
@pytest.mark.parametrize("kind", ["all", "upper", "random"])
def test_closing_exchange_matches_oracle(emu, kind, n, dtype):
    rng = np.random.default_rng(n)
    init = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    init /= np.linalg.norm(init)
    gates = swaps(n, kind)
    st = init.copy()
    plan(emu, n, gates, dtype, st)
    o = OracleState(n)
    o.set_state(init)
    o.apply(gates)
    assert np.abs(st - o.state()).max() < TOL[dtype]


@pytest.mark.parametrize("n,gates,dtype,most", [
    (20, lambda: circuits.random_layers(20, 20, 20240601), C128, 14),
    (32, lambda: circuits.random_layers(32, 16, 20240601, iswap_frac=0.1), C64, 24),
    (28, lambda: circuits.qft(28), C64, 4),
    (28, lambda: circuits.qft(28), C128, 4),
])
def test_benchmark_circuits_run_in_few_passes(emu, n, gates, dtype, most):
    assert plan(emu, n, gates(), dtype)[0] <= most


def phase_estimation(n):
    """Phase estimation of a phase gate on the highest qubit with n - 1 counting
    qubits, textbook form: 2^k controlled phases from counting qubit k, so that
    2^(n-1) - 1 phases share a hub, then the inverse QFT of the counting qubits."""
    t = n - 1
    spec = [("X", (t,))] + [("H", (k,)) for k in range(t)]
    spec += [("CR", (k, t), 0.7) for k in range(t) for _ in range(1 << k)]
    for j in reversed(range(t)):
        spec += [("H", (j,))] + [("CR", (j, i), -np.pi / 2 ** (j - i)) for i in range(j)]
    return circuits.make_gates(spec)


def phases_on(n, hubs, count):
    """`count` phases on each hub, the partners in turn, then an H on it."""
    spec = []
    for h in hubs:
        others = [q for q in range(n) if q != h]
        spec += [("CR", (h, others[k % len(others)]), 0.1 + 0.01 * k) for k in range(count)] + [("H", (h,))]
    return circuits.make_gates(spec)


# lists whose phases on one hub outnumber a parameter block's entries
MANY_PHASES = {
    "estimation10": (10, lambda: phase_estimation(10)),
    "estimation13": (13, lambda: phase_estimation(13)),
    "hub300": (12, lambda: phases_on(12, [0], 300)),
    "hub257": (10, lambda: phases_on(10, [0], 257)),
    "hubs": (13, lambda: phases_on(13, [0, 12, 5], 300)),
    "pair300": (9, lambda: circuits.make_gates([("CR", (2, 7), 0.3 + 0.01 * k) for k in range(300)] + [("H", (2,)), ("H", (7,))])),
}


@pytest.mark.parametrize("dtype", [C64, C128])
@pytest.mark.parametrize("kind", list(MANY_PHASES))
def test_many_phases_on_one_hub(emu, kind, dtype):
    n, gates = MANY_PHASES[kind][0], MANY_PHASES[kind][1]()
    rng = np.random.default_rng(n)
    init = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    init /= np.linalg.norm(init)
    st = init.copy()
    plan(emu, n, gates, dtype, st)
    o = OracleState(n)
    o.set_state(init)
    o.apply(gates)
    # FP64: two roundings of 1.1e-16 per gate on either side; FP32: phases on a
    # hub are multiplied in FP64, so that their number does not show
    assert np.abs(st - o.state()).max() < (TOL[C64] if dtype == C64 else 4.5e-16 * len(gates))


def idle(n, layers):
    """Layers that leave the highest qubit alone until the last gate."""
    return np.concatenate([circuits.random_layers(n - 1, layers, n), circuits.make_gates([("H", (n - 1,))])])


@pytest.mark.parametrize("dtype", [C64, C128])
@pytest.mark.parametrize("n", [9, 13])
@pytest.mark.parametrize("kind", ["layers", "idle"])
def test_lists_past_the_planning_window(emu, kind, n, dtype):
    """More gates than the planner looks at at once and than a pass is handed."""
    layers = 3000 // (n + n // 2)
    gates = circuits.random_layers(n, layers, n) if kind == "layers" else idle(n, layers)
    rng = np.random.default_rng(n)
    init = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    init /= np.linalg.norm(init)
    st = init.copy()
    plan(emu, n, gates, dtype, st)
    o = OracleState(n)
    o.set_state(init)
    o.apply(gates)
    # as above: per gate two roundings on either side, FP32 as TOL for its 150 gates
    assert np.abs(st - o.state()).max() < (TOL[C64] / 150 if dtype == C64 else 4.5e-16) * len(gates)


@pytest.mark.parametrize("n,kind", [(9, "layers"), (12, "layers"), (20, "layers"), (20, "idle")])
def test_planning_time_is_linear(emu, n, kind):
    """Time per gate of 60,000 gates stays near that of 2,000 (copies of the
    rest of the list in every pass made it ten times as long)."""
    def per_gate(count):
        layers = 2000 // (n + n // 2)
        one = circuits.random_layers(n, layers, n) if kind == "layers" else idle(n, layers)
        gates = np.tile(one, max(1, count // len(one)))
        best = 1e9
        for _ in range(3):
            t = time.process_time()
            plan(emu, n, gates, C64)
            best = min(best, time.process_time() - t)
        return best / len(gates)

    assert per_gate(60000) < 3 * per_gate(2000)


def gate_by_gate(init, gates, dtype):
    """RX, RY, RZ, H, CNOT, CR and SWAP records on a state of `dtype`, one by one,
    with the gates' FP64 matrices."""
    x = init.astype(dtype)
    for g in gates:
        op, t, q = int(g["op"]), float(g["theta"]) / 2, [int(k) for k in g["q"]]
        if op in (OP["CR"], OP["SWAP"]):
            i = np.arange(len(x))
            if op == OP["CR"]:
                i = i[(i >> q[0] & 1 == 1) & (i >> q[1] & 1 == 1)]
                x[i] *= dtype(np.cos(2 * t) + 1j * np.sin(2 * t))
            else:
                i = i[(i >> q[0] & 1 == 1) & (i >> q[1] & 1 == 0)]
                k = i ^ (1 << q[0] | 1 << q[1])
                x[i], x[k] = x[k], x[i]
            continue
        if op == OP["CNOT"]:
            i = np.arange(len(x))
            i = i[(i >> q[0] & 1 == 1) & (i >> q[1] & 1 == 0)]
            x[i], x[i | 1 << q[1]] = x[i | 1 << q[1]], x[i]
            continue
        c, s, h = np.cos(t), np.sin(t), 0.707106781186548
        m = {OP["RX"]: [[c, -1j * s], [-1j * s, c]], OP["RY"]: [[c, -s], [s, c]],
             OP["RZ"]: [[c - 1j * s, 0], [0, c + 1j * s]], OP["H"]: [[h, h], [h, -h]]}[op]
        v = x.reshape(-1, 2, 1 << q[0])
        a, b = v[:, 0].copy(), v[:, 1].copy()
        v[:, 0] = dtype(m[0][0]) * a + dtype(m[0][1]) * b
        v[:, 1] = dtype(m[1][0]) * a + dtype(m[1][1]) * b
    return x


@pytest.mark.parametrize("n,layers", [(9, 8), (12, 20), (10, 60)])
def test_complex128_is_as_exact_as_gate_by_gate(emu, n, layers):
    """Against extended precision: the pivots, ratios and phases that a pass rounds
    must not add up over its gates, in the norm or in the state."""
    drift, err, plain, passes = [], [], [], 0
    for seed in range(12):
        rng = np.random.default_rng(seed)
        init = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
        init /= np.linalg.norm(init)
        gates = circuits.random_layers(n, layers, seed)
        st = init.copy()
        passes = max(passes, plan(emu, n, gates, C128, st)[0])
        exact = gate_by_gate(init, gates, np.clongdouble)
        norm = np.sqrt((np.abs(exact) ** 2).sum())
        drift.append(float(np.sqrt((np.abs(st.astype(np.clongdouble)) ** 2).sum()) - norm))
        err.append(float(np.sqrt((np.abs(st - exact) ** 2).sum())))
        plain.append(float(np.sqrt((np.abs(gate_by_gate(init, gates, np.complex128) - exact) ** 2).sum())))
    # one rounding of a pass's factor (1.1e-16), and 1e-16 for the phases, whose
    # rounding is split between the halves of the state
    assert np.sqrt(np.mean(np.square(drift))) < 1.1e-16 * passes + 1e-16
    assert np.mean(err) < np.mean(plain)


def test_factors_of_passes_do_not_drift(emu):
    """The factor of each pass is rounded; the next pass makes up for it.  A QFT's
    passes have the square roots of its H gates as factors: over all of them the
    norm is off by one rounding at most."""
    n = 13
    gates = circuits.qft(n)
    for seed in range(4):
        rng = np.random.default_rng(seed)
        init = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
        init /= np.linalg.norm(init)
        st = init.copy()
        assert plan(emu, n, gates, C128, st)[0] > 1
        exact = gate_by_gate(init, gates, np.clongdouble)
        norms = [np.sqrt((np.abs(v.astype(np.clongdouble)) ** 2).sum()) for v in (st, exact)]
        assert abs(float(norms[0] - norms[1])) < 1.1e-16
