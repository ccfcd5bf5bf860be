"""The staged passes (k_stage) against the oracle: the narrowest states they
take, one tile, the first states of several tiles, parameter blocks of both
sizes, and lists that stay on the per-gate kernels."""
import numpy as np
import pytest

from oracle.pyoracle import OracleState
from qpanda_b200 import StateVector, circuits
from tests.test_stage_emulation import LISTS

pytestmark = pytest.mark.gpu

TOL = {"c64": 1e-5, "c128": 1e-12}


def random_state(n, seed):
    rng = np.random.default_rng(seed)
    v = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    return v / np.linalg.norm(v)


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n", [8, 9, 11, 12, 13, 17])
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
