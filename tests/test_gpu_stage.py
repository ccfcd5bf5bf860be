"""The staged passes (k_stage) against the oracle: the narrowest states they
take, one tile, the first states of several tiles, parameter blocks of both
sizes, and lists that stay on the per-gate kernels."""
import ctypes as C
import time

import numpy as np
import pytest

from oracle.pyoracle import OracleState
from qpanda_b200 import Server, StateVector, circuits
from qpanda_b200.capi import check, lib
from tests.test_stage_emulation import LISTS, MANY_PHASES, swaps

pytestmark = pytest.mark.gpu

TOL = {"c64": 1e-5, "c128": 1e-12}


def random_state(n, seed):
    rng = np.random.default_rng(seed)
    v = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    return v / np.linalg.norm(v)


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n", [7, 8, 9, 11, 12, 13, 17])
@pytest.mark.parametrize("kind", list(LISTS))
def test_lists_match_oracle(need_gpu, kind, n, dtype):
    init, gates = random_state(n, n), LISTS[kind](n)
    with StateVector(n, dtype) as sv:
        sv.set_state(init.astype(np.complex64) if dtype == "c64" else init)
        sv.apply(gates)
        got = sv.get_state()
    o = OracleState(n)
    o.set_state(init)
    o.apply(gates)
    assert np.abs(got - o.state()).max() < TOL[dtype]


@pytest.mark.parametrize("dtype", ["c64", "c128"])
def test_wide_states(need_gpu, dtype):
    """23 and 24 qubits: tiles on the highest qubits, a lone gate, two phases
    that the per-gate kernels keep."""
    for n, gates in ((23, circuits.random_layers(23, 2, 5, iswap_frac=0.2)), (24, circuits.qft(24)[-40:]),
                     (24, circuits.make_gates([("CR", (22, 23), 0.5), ("CR", (21, 20), 0.25)])),
                     (23, circuits.make_gates([("RY", (22,), 1.0)]))):
        init = random_state(n, n)
        with StateVector(n, dtype) as sv:
            sv.set_state(init.astype(np.complex64) if dtype == "c64" else init)
            sv.apply(gates)
            got = sv.get_state()
        o = OracleState(n)
        o.set_state(init)
        o.apply(gates)
        assert np.abs(got - o.state()).max() < TOL[dtype]


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n", [12, 13, 16])
def test_lists_from_zero_state(need_gpu, n, dtype):
    """From |0...0> the first passes leave tiles of zeros alone; amplitudes that
    the caller has put into the state since, through its device address, are
    no zeros and take part."""
    import torch

    gates = circuits.random_layers(n, 3, n, iswap_frac=0.2)
    for put in (False, True):
        with StateVector(n, dtype) as sv:
            sv.apply(circuits.random_layers(n, 1, 1))
            sv.reset()
            init = np.zeros(1 << n, complex)
            init[0] = 1
            if put:
                p = C.c_void_p()
                check(lib().qs_device_ptr(sv.handle, C.byref(p)))
                mem = type("Mem", (), {"__cuda_array_interface__": {
                    "shape": (1 << n,), "typestr": "<c8" if dtype == "c64" else "<c16", "data": (p.value, False),
                    "version": 2}})()
                torch.as_tensor(mem, device="cuda")[(1 << n) - 3] = 0.5
                init[-3] = 0.5
            sv.apply(gates)
            got = sv.get_state()
        o = OracleState(n)
        o.set_state(init)
        o.apply(gates)
        assert np.abs(got - o.state()).max() < TOL[dtype]


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n", [13, 16, 19])
@pytest.mark.parametrize("kind", ["all", "upper", "random"])
def test_closing_exchange(need_gpu, kind, n, dtype):
    init, gates = random_state(n, n), swaps(n, kind)
    with StateVector(n, dtype) as sv:
        sv.set_state(init.astype(np.complex64) if dtype == "c64" else init)
        sv.apply(gates)
        got = sv.get_state()
    o = OracleState(n)
    o.set_state(init)
    o.apply(gates)
    assert np.abs(got - o.state()).max() < TOL[dtype]


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("kind", list(MANY_PHASES))
def test_many_phases_on_one_hub(need_gpu, kind, dtype):
    n, gates = MANY_PHASES[kind][0], MANY_PHASES[kind][1]()
    init = random_state(n, n)
    with StateVector(n, dtype) as sv:
        sv.set_state(init.astype(np.complex64) if dtype == "c64" else init)
        sv.apply(gates)
        got = sv.get_state()
    o = OracleState(n)
    o.set_state(init)
    o.apply(gates)
    # FP64: two roundings of 1.1e-16 per gate on either side
    assert np.abs(got - o.state()).max() < max(TOL[dtype], 4.5e-16 * len(gates))


def test_many_phases_on_one_hub_served(need_gpu):
    """The same through the serving loop, below the width of its plans."""
    n, gates = MANY_PHASES["estimation10"][0], MANY_PHASES["estimation10"][1]()
    srv = Server(slots=1)
    rid = srv.submit(n, gates, "probs")
    srv.wait(rid)
    o = OracleState(n)
    o.apply(gates)
    assert np.abs(srv.fetch_probs(rid) - o.probs()).max() < 1e-5
    srv.release(rid)
    srv.close()


def ladder(n):
    return circuits.make_gates([("CR", (0, q), 0.1 * q) for q in range(1, n)])


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n", [8, 11, 12, 13, 16, 23])
def test_lone_ladder(need_gpu, n, dtype):
    init, gates = random_state(n, n), ladder(n)
    with StateVector(n, dtype) as sv:
        sv.set_state(init.astype(np.complex64) if dtype == "c64" else init)
        sv.apply(gates)
        got = sv.get_state()
    o = OracleState(n)
    o.set_state(init)
    o.apply(gates)
    assert np.abs(got - o.state()).max() < TOL[dtype]


@pytest.mark.parametrize("dtype", ["c64", "c128"])
def test_lone_ladder_is_one_pass(need_gpu, dtype):
    """A list that joins into one ladder takes one read and write of the state,
    not a launch per phase (23 phases of a quarter of the state or more)."""
    import torch

    n, gates = 24, ladder(24)
    with StateVector(n, dtype) as sv:
        def best(f):
            times = []
            for _ in range(10):
                torch.cuda.synchronize()
                t = time.perf_counter()
                f()
                torch.cuda.synchronize()
                times.append(time.perf_counter() - t)
            return min(times)

        def one_by_one():
            for k in range(len(gates)):
                check(lib().qs_gate_apply(sv.handle, C.c_void_p(gates[k:k + 1].ctypes.data)))

        assert best(lambda: sv.apply(gates)) < 0.6 * best(one_by_one)
