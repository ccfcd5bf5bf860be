"""The work whose speed is measured, case by case, through the package's public entry points.

listed() names the cases, draw() gives more of the same ranges, prepare() makes what a
program has in hand before the call (states, gate records, plans, a server), run() makes one
pass and work() counts what a pass cannot do without.  exact() gives the same outputs in 64
bits from plain torch operations on the gate definitions restated below.

States are handed out where they lie, as torch views of their device memory.  Values that are
computed from a complex64 state (probabilities, expectations) are handed out in 32 bits, the
precision that such a state carries; from a complex128 state in 64.
"""
import ctypes
import math
import random

import numpy as np
import torch

from qpanda_b200 import Batch, FusionPlan, StateVector, circuits
from qpanda_b200.capi import Server, check, lib


def listed():
    return [
        # A small program run to the end: the shape of the command-line and teaching programs,
        # where launches and host work count.
        {"name": "circuit_9q_c128", "kind": "circuit", "n": 9, "depth": 8, "dtype": "c128", "iswap": 0.0, "shots": 256},
        # The 20-qubit random circuit with its probability vector and shots, double precision.
        {"name": "circuit_20q_c128", "kind": "circuit", "n": 20, "depth": 20, "dtype": "c128", "iswap": 0.0, "shots": 1024},
        # A large single-precision circuit, gate list in, state left on the device.
        {"name": "circuit_30q_c64", "kind": "circuit", "n": 30, "depth": 16, "dtype": "c64", "iswap": 0.1, "shots": 0},
        # The QFT of a state in hand, in both precisions, at an even and an odd width.
        {"name": "qft_28q_c64", "kind": "qft", "n": 28, "dtype": "c64"},
        {"name": "qft_27q_c128", "kind": "qft", "n": 27, "dtype": "c128"},
        # A host program that sends matrices one call at a time (any qubits, with controls).
        {"name": "unitaries_24q_c64", "kind": "unitaries", "n": 24, "calls": 48, "dtype": "c64"},
        # Fused plans kept by the program: the large circuit with the second buffer, and a
        # middle-sized one in place.
        {"name": "fused_30q_c64", "kind": "fused", "n": 30, "depth": 16, "iswap": 0.1, "remap": 1},
        {"name": "fused_21q_c64", "kind": "fused", "n": 21, "depth": 16, "iswap": 0.0, "remap": 0},
        # A variational sweep in one launch: uneven widths and depths, all <Z_i Z_i+1> back.
        {"name": "sweep_256", "kind": "sweep", "circuits": 256, "qmin": 10, "qmax": 22, "lmin": 4, "lmax": 12},
        # Layers with measurements between them, measured qubits reset, marginals at the end.
        {"name": "midmeasure_26q_c64", "kind": "midmeasure", "n": 26, "rounds": 3, "per_round": 2, "bins": 10, "dtype": "c64"},
        # Shots and a marginal of a state in hand.
        {"name": "shots_27q_c64", "kind": "shots", "n": 27, "shots": 1024, "bins": 16, "dtype": "c64"},
        # A burst of requests to the serving loop, narrow and wide, shots and probabilities.
        {"name": "requests_24", "kind": "requests", "requests": 24, "qmin": 8, "qmax": 20, "dmin": 4, "dmax": 32},
    ]


def draw(rng):
    kind = rng.choice(["circuit", "circuit", "qft", "unitaries", "fused", "sweep", "midmeasure", "shots", "requests"])
    dtype = rng.choice(["c64", "c128"])
    most = 30 if dtype == "c64" else 28
    if kind == "circuit":
        n = rng.randint(4, most)
        # shots where their bits do not hang on the last bit of a single-precision sum
        return {"kind": kind, "n": n, "depth": rng.randint(2, 16), "dtype": dtype, "iswap": rng.choice([0.0, 0.1]),
                "shots": rng.randint(1, 1024) if dtype == "c128" and n <= 22 else 0}
    if kind == "qft":
        return {"kind": kind, "n": rng.randint(5, most), "dtype": dtype}
    if kind == "unitaries":
        return {"kind": kind, "n": rng.randint(8, most - 2), "calls": rng.randint(16, 64), "dtype": dtype}
    if kind == "fused":
        n = rng.randint(12, 30)
        return {"kind": kind, "n": n, "depth": rng.randint(4, 16), "iswap": rng.choice([0.0, 0.1]),
                "remap": rng.choice([0, 1]) if n >= 20 else 0}
    if kind == "sweep":
        qmin = rng.randint(4, 16)
        lmin = rng.randint(2, 8)
        return {"kind": kind, "circuits": int(16 * 2 ** rng.uniform(0, 4)), "qmin": qmin, "qmax": rng.randint(qmin, 22),
                "lmin": lmin, "lmax": rng.randint(lmin, 12)}
    if kind == "midmeasure":
        n = rng.randint(8, most - 2)
        return {"kind": kind, "n": n, "rounds": rng.randint(1, 4), "per_round": rng.randint(1, 3),
                "bins": rng.randint(1, 8), "dtype": dtype}
    if kind == "shots":
        n = rng.randint(8, most - 1)
        return {"kind": kind, "n": n, "shots": int(2 ** rng.uniform(0, 11)), "bins": rng.randint(1, min(n, 18)), "dtype": dtype}
    qmin = rng.randint(5, 14)
    return {"kind": kind, "requests": rng.randint(8, 24), "qmin": qmin, "qmax": rng.randint(qmin, 20), "dmin": 4,
            "dmax": rng.randint(5, 32)}


# ---------------------------------------------------------------- inputs: (operation, qubits, angle)

def _layers(n, depth, rng, iswap=0.0):
    """Per layer an RX, RY or RZ on every qubit, then CNOT (or iSWAP) on a random perfect matching."""
    spec = []
    for _ in range(depth):
        for q in range(n):
            spec.append((rng.choice(("RX", "RY", "RZ")), (q,), rng.uniform(0.0, 2 * math.pi)))
        order = list(range(n))
        rng.shuffle(order)
        for p in range(n // 2):
            spec.append(("ISWAP" if rng.random() < iswap else "CNOT", (order[2 * p], order[2 * p + 1])))
    return spec


def _ansatz(n, layers, rng):
    """Per layer RY then RZ on every qubit, then a CNOT ladder."""
    spec = []
    for _ in range(layers):
        for op in ("RY", "RZ"):
            spec += [(op, (q,), rng.uniform(0.0, 2 * math.pi)) for q in range(n)]
        spec += [("CNOT", (q, q + 1)) for q in range(n - 1)]
    return spec


def _qft(n):
    spec = []
    for j in range(n):
        spec += [("CR", (j, i), math.pi / 2 ** (j - i)) for i in range(j)]
        spec.append(("H", (j,)))
    return spec + [("SWAP", (k, n - 1 - k)) for k in range(n // 2)]


def _unitary(rng, d):
    m = np.array([[complex(rng.gauss(0, 1), rng.gauss(0, 1)) for _ in range(d)] for _ in range(d)])
    return np.linalg.qr(m)[0]


def _unitaries(n, calls, rng):
    """(call, qubits, matrix or phase, control mask), on any qubits, one in three with controls."""
    out = []
    for _ in range(calls):
        qs = rng.sample(range(n), 4)
        what = rng.choice(["1q", "1q", "2q", "exchange", "phase"])
        used = {"1q": 1, "2q": 2, "exchange": 2, "phase": 0}[what]
        ctrl = sum(1 << q for q in qs[used:used + rng.choice([0, 0, 1, 2])][:4 - used])
        if what == "phase":
            a = rng.uniform(0, 2 * math.pi)
            out.append((what, (), complex(math.cos(a), math.sin(a)), sum(1 << q for q in qs[:rng.choice([1, 2, 2, 3])])))
        else:
            out.append((what, tuple(qs[:used]), _unitary(rng, 4 if what == "2q" else 2), ctrl))
    return out


def _sizes(case, count, a, b):
    """`count` pairs of whole numbers between case[a + "min"] and case[a + "max"], and b's: the case's own, whatever the seed."""
    rng = random.Random(str(sorted((k, v) for k, v in case.items() if k != "name")))
    return [(rng.randint(case[a + "min"], case[a + "max"]), rng.randint(case[b + "min"], case[b + "max"])) for _ in range(count)]


def _sweep(case, rng):
    return [(n, _ansatz(n, layers, rng)) for n, layers in _sizes(case, case["circuits"], "q", "l")]


def _midmeasure(case, rng):
    n = case["n"]
    rounds = [(_layers(n, 1, rng), [(q, rng.random()) for q in rng.sample(range(n), case["per_round"])])
              for _ in range(case["rounds"])]
    return rounds, rng.sample(range(n), case["bins"])


def _requests(case, rng):
    return [(n, _layers(n, depth, rng), "probs" if k % 2 else "shots", rng.randrange(1 << 31))
            for k, (n, depth) in enumerate(_sizes(case, case["requests"], "q", "d"))]


def _gaussian(n, seed, dtype):
    """A normalised state of i.i.d. complex Gaussian amplitudes."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn(1 << n, 2, dtype=torch.float32 if dtype == "c64" else torch.float64, device="cuda", generator=g)
    x /= torch.linalg.vector_norm(x, dtype=torch.float64)
    return torch.view_as_complex(x)


class _Memory:
    """A state's amplitudes as an array on the device."""

    def __init__(self, sv):
        p = ctypes.c_void_p()
        check(lib().qs_device_ptr(sv.handle, ctypes.byref(p)))
        self.sv = sv
        self.__cuda_array_interface__ = {"shape": (1 << sv.n,), "typestr": "<c8" if sv.dtype == 0 else "<c16",
                                         "data": (p.value, False), "version": 2}


def _view(sv):
    return torch.as_tensor(_Memory(sv), device="cuda")


# ---------------------------------------------------------------- prepare and run

def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "sweep":
        s["batch"] = Batch([(n, circuits.make_gates(spec)) for n, spec in _sweep(case, rng)])
        return s
    if kind == "requests":
        s["requests"] = [(n, circuits.make_gates(spec), what, np.random.default_rng(us).uniform(size=(256, n)))
                         for n, spec, what, us in _requests(case, rng)]
        s["server"] = Server()
        return s
    n, dtype = case["n"], case.get("dtype", "c64")
    sv = s["state"] = StateVector(n, dtype)
    s["view"] = _view(sv)
    if kind == "circuit":
        s["gates"] = circuits.make_gates(_layers(n, case["depth"], rng, case["iswap"]))
        s["uniforms"] = np.random.default_rng(seed).uniform(size=(case["shots"], n))
    elif kind == "fused":
        s["plan"] = FusionPlan(n, circuits.make_gates(_layers(n, case["depth"], rng, case["iswap"])), remap=case["remap"])
    elif kind == "midmeasure":
        rounds, s["bins"] = _midmeasure(case, rng)
        s["rounds"] = [(circuits.make_gates(spec), measured) for spec, measured in rounds]
        s["flip"] = [circuits.make_gates([("X", (q,))]) for q in range(n)]
    else:
        s["view"].copy_(_gaussian(n, seed, dtype))
        if kind == "qft":
            s["gates"] = circuits.make_gates(_qft(n))
        elif kind == "unitaries":
            s["calls"] = _unitaries(n, case["calls"], rng)
        elif kind == "shots":
            s["uniforms"] = np.random.default_rng(seed).uniform(size=(case["shots"], n))
            s["bins"] = rng.sample(range(n), case["bins"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "sweep":
        s["batch"].run()
        return np.concatenate(s["batch"].zz()).astype(np.float32)
    if kind == "requests":
        return _run_requests(s)
    sv = s["state"]
    if kind == "circuit":
        sv.reset()
        sv.apply(s["gates"])
        if not len(s["uniforms"]):
            return s["view"]
        return s["view"], sv.probs(), sv.sample(range(sv.n), s["uniforms"]).astype(np.int64)
    if kind == "qft":
        sv.apply(s["gates"])
        return s["view"]
    if kind == "unitaries":
        for what, q, m, ctrl in s["calls"]:
            if what == "1q":
                sv.apply_1q(q[0], m, ctrl)
            elif what == "2q":
                sv.apply_2q(q[0], q[1], m, ctrl)
            elif what == "exchange":
                sv.apply_exchange(q[0], q[1], m, ctrl)
            else:
                sv.apply_phase(ctrl, m)
        return s["view"]
    if kind == "fused":
        sv.reset()
        s["plan"].apply(sv)
        return s["view"]
    if kind == "midmeasure":
        sv.reset()
        got = []
        for gates, measured in s["rounds"]:
            sv.apply(gates)
            for q, u in measured:
                got.append(sv.measure(q, u))
                if got[-1]:
                    sv.apply(s["flip"][q])
        probs = np.append(sv.probs(s["bins"]), sv.prob_zero(s["bins"][0]))
        return s["view"], np.array(got), probs.astype(np.float32) if sv.dtype == 0 else probs
    probs = sv.probs(s["bins"])
    return sv.sample(range(sv.n), s["uniforms"]).astype(np.int64), probs.astype(np.float32) if sv.dtype == 0 else probs


def _run_requests(s):
    srv = s["server"]
    ids = [srv.submit(n, gates, what, u if what == "shots" else None) for n, gates, what, u in s["requests"]]
    shots, probs = [], []
    for rid, (n, gates, what, u) in zip(ids, s["requests"]):
        srv.wait(rid)
        if what == "shots":
            shots.append(srv.shots(rid))
        else:
            probs.append(srv.fetch_probs(rid).astype(np.float32))
        srv.release(rid)
    return np.concatenate(shots).astype(np.int64), np.concatenate(probs)


# ---------------------------------------------------------------- what a pass cannot do without

#: floating-point operations for each amplitude that a gate changes (complex multiply 6, add 2;
#: matrices with real and imaginary entries only need half of it)
_FLOPS = {"RX": 6, "RY": 6, "RZ": 6, "H": 4, "CR": 6, "CNOT": 0, "ISWAP": 0, "SWAP": 0}


def _flops(n, spec):
    return sum(_FLOPS[g[0]] * (1 << n) / (4 if g[0] == "CR" else 1) for g in spec)


def work(case):
    kind, rng = case["kind"], random.Random(1)
    if kind == "sweep":
        got = _sweep(case, rng)
        return {"bytes": sum(8.0 * n for n, _ in got), "flops": sum(_flops(n, spec) for n, spec in got)}
    if kind == "requests":
        got = _requests(case, rng)
        return {"bytes": sum((8.0 * 256 * (n + 1) if what == "shots" else 8.0 * (1 << n)) for n, _, what, _ in got),
                "flops": sum(_flops(n, spec) for n, spec, _, _ in got)}
    n, state = case["n"], float((16 if case.get("dtype") == "c128" else 8) << case["n"])
    if kind == "circuit":       # the state written, its probabilities read off, the uniforms read, the shots written
        more = state + 8.0 * (1 << n) + 8.0 * case["shots"] * (n + 1) if case["shots"] else 0.0
        return {"bytes": state + more, "flops": _flops(n, _layers(n, case["depth"], rng, case["iswap"]))}
    if kind == "fused":
        return {"bytes": state, "flops": _flops(n, _layers(n, case["depth"], rng, case["iswap"]))}
    if kind == "qft":
        return {"bytes": 2 * state, "flops": _flops(n, _qft(n))}
    if kind == "unitaries":     # each call is one of its own: the amplitudes that it changes, read and written
        moved = flops = 0.0
        for what, q, _, ctrl in _unitaries(n, case["calls"], rng):
            part = 0.5 ** bin(ctrl).count("1") * (0.5 if what == "exchange" else 1.0)
            moved += 2 * state * part
            flops += (1 << n) * part * {"1q": 14, "exchange": 14, "2q": 30, "phase": 6}[what]
        return {"bytes": moved, "flops": flops}
    if kind == "midmeasure":    # each measurement reads what is there and writes the collapsed state
        m = case["rounds"] * case["per_round"]
        return {"bytes": state * (case["rounds"] + 2 * m + 2), "flops": case["rounds"] * n * 6.0 * (1 << n)}
    return {"bytes": 2 * state + 8.0 * (1 << case["bins"]) + 8.0 * case["shots"] * (n + 1), "flops": 2 * 4.0 * (1 << n)}


# ---------------------------------------------------------------- the same in 64 bits

_SQ2 = 0.707106781186548        # as the gate definitions have it


def _matrix(op, t):
    c, s = math.cos(t / 2), math.sin(t / 2)
    return np.array({"H": [[_SQ2, _SQ2], [_SQ2, -_SQ2]], "X": [[0, 1], [1, 0]], "RX": [[c, -1j * s], [-1j * s, c]],
                     "RY": [[c, -s], [s, c]], "RZ": [[c - 1j * s, 0], [0, c + 1j * s]]}[op], dtype=complex)


class _Exact:
    """A complex128 state under plain torch operations; 1-qubit gates wait and are applied five qubits at a time."""

    def __init__(self, n, x=None):
        self.n = n
        self.x = torch.zeros(1 << n, dtype=torch.complex128, device="cuda") if x is None else x.to(torch.complex128)
        if x is None:
            self.x[0] = 1
        self.waiting = {}

    def part(self, bits):
        """The amplitudes whose qubits have these values ({qubit: 0 or 1})."""
        shape, at, top = [], [], self.n
        for q in sorted(bits, reverse=True):
            shape += [1 << (top - q - 1), 2]
            at += [slice(None), bits[q]]
            top = q
        return self.x.view(shape + [1 << top])[tuple(at + [slice(None)])]

    def flush(self):
        for low in range(0, self.n, 5):
            qs = [q for q in range(low, min(low + 5, self.n)) if q in self.waiting]
            if len(qs) > 1:
                k = min(5, self.n - low)
                m = np.eye(1)
                for q in range(low, low + k):
                    m = np.kron(self.waiting.get(q, np.eye(2)), m)
                m = torch.from_numpy(m).to("cuda")
                if low == 0:
                    self.x = (self.x.view(-1, 1 << k) @ m.T).view(-1)
                else:
                    self.x = torch.matmul(m, self.x.view(-1, 1 << k, 1 << low)).reshape(-1)
            elif qs:
                self.dense(qs, self.waiting[qs[0]], 0)
        self.waiting = {}

    def dense(self, qs, m, ctrl):
        """A matrix on the qubits qs (index bit j = qubit qs[j]) where every control bit is set."""
        on = {q: 1 for q in range(self.n) if ctrl >> q & 1}
        parts = [self.part({**on, **{q: b >> j & 1 for j, q in enumerate(qs)}}) for b in range(1 << len(qs))]
        old = [p.clone() for p in parts]
        for p, row in zip(parts, m):
            p.zero_()
            for o, v in zip(old, row):
                if v != 0:
                    p.add_(o, alpha=complex(v))

    def exchange(self, a, b, m, ctrl):
        on = {q: 1 for q in range(self.n) if ctrl >> q & 1}
        x, y = self.part({**on, a: 1, b: 0}), self.part({**on, a: 0, b: 1})
        if m is None:
            t = x.clone()
            x.copy_(y)
            y.copy_(t)
        else:
            t = complex(m[0][0]) * x + complex(m[0][1]) * y
            y.copy_(complex(m[1][0]) * x + complex(m[1][1]) * y)
            x.copy_(t)

    def gate(self, op, q, t=0.0):
        if op in ("H", "X", "RX", "RY", "RZ"):
            self.waiting[q[0]] = _matrix(op, t) @ self.waiting.get(q[0], np.eye(2))
            return
        if any(k in self.waiting for k in q):
            self.flush()
        if op == "CNOT":
            x, y = self.part({q[0]: 1, q[1]: 0}), self.part({q[0]: 1, q[1]: 1})
            t = x.clone()
            x.copy_(y)
            y.copy_(t)
        elif op == "CR":
            self.part({q[0]: 1, q[1]: 1}).mul_(complex(math.cos(t), math.sin(t)))
        else:
            self.exchange(q[0], q[1], None if op == "SWAP" else [[0, 1j], [1j, 0]], 0)

    def gates(self, spec):
        for g in spec:
            self.gate(*g)
        self.flush()
        return self

    def probs(self, qubits):
        """Marginal over the qubits, index bit j = qubits[j]."""
        p = self.x.real.square() + self.x.imag.square()
        kept = sorted(qubits, reverse=True)
        shape, top = [], self.n
        for q in kept:
            shape += [1 << (top - q - 1), 2]
            top = q
        p = p.view(shape + [1 << top])
        p = p.sum(dim=[d for d in range(p.dim()) if d % 2 == 0])
        return p.permute([kept.index(q) for q in reversed(qubits)]).reshape(-1)


def exact(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "sweep":
        out = []
        for n, spec in _sweep(case, rng):
            e = _Exact(n).gates(spec)
            pairs = [e.probs([i, i + 1]) for i in range(n - 1)]
            out.append(torch.stack(pairs) @ torch.tensor([1.0, -1.0, -1.0, 1.0], dtype=torch.float64, device="cuda"))
        return torch.cat(out).cpu().numpy()
    if kind == "requests":
        got = [_Exact(n).gates(spec).probs(list(range(n))) for n, spec, what, _ in _requests(case, rng) if what == "probs"]
        return None, torch.cat(got).cpu().numpy()
    n, dtype = case["n"], case.get("dtype", "c64")
    if kind in ("circuit", "fused"):
        e = _Exact(n).gates(_layers(n, case["depth"], rng, case["iswap"]))
        return (e.x, e.probs(list(range(n))), None) if case.get("shots") else e.x
    if kind == "midmeasure":
        rounds, bins = _midmeasure(case, rng)
        e = _Exact(n)
        for spec, measured in rounds:
            e.gates(spec)
            for q, u in measured:
                p0 = float(e.probs([q])[0])
                got = int(float(np.float32(u)) > p0)
                e.part({q: 1 - got}).zero_()
                e.x *= 1 / math.sqrt(1 - p0 if got else p0)
                if got:
                    e.gates([("X", (q,))])
        probs = torch.cat([e.probs(bins), e.probs(bins[:1])[:1]])
        return e.x, None, probs.cpu().numpy()
    e = _Exact(n, _gaussian(n, seed, dtype))
    if kind == "qft":
        return e.gates(_qft(n)).x
    if kind == "unitaries":
        for what, q, m, ctrl in _unitaries(n, case["calls"], rng):
            if what in ("1q", "2q"):
                e.dense(list(q), m, ctrl)
            elif what == "exchange":
                e.exchange(q[0], q[1], m, ctrl)
            else:
                e.part({k: 1 for k in range(n) if ctrl >> k & 1}).mul_(m)
        return e.x
    return None, e.probs(rng.sample(range(n), case["bins"])).cpu().numpy()
