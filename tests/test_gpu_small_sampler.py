"""The one-CTA sampler of narrow states (up to 11 qubits) against the oracle's
literal per-shot re-measurement, and small marginals that land in the state's
pinned host buffer: widths on both sides of the limits, subsets in any order,
shots on both sides of the buffer's size."""
import time

import numpy as np
import pytest

from oracle.pyoracle import OracleState
from qpanda_b200 import StateVector, circuits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n,shots", [(1, 3), (2, 1), (5, 40), (9, 512), (9, 513), (11, 700), (12, 64)])
def test_shots_and_marginals(need_gpu, n, shots, dtype):
    rng = np.random.default_rng(100 * n + shots)
    gates = circuits.random_layers(n, 3, n) if n > 1 else circuits.make_gates([("RY", (0,), 0.8)])
    o = OracleState(n)
    o.apply(gates)
    st = o.state()
    if dtype == "c64":                       # the oracle on the amplitudes that the state holds
        st = st.astype(np.complex64).astype(np.complex128)
        o.set_state(st)
    with StateVector(n, dtype) as sv:
        sv.set_state(st.astype(np.complex64) if dtype == "c64" else st)
        for m in sorted({1, (n + 1) // 2, n}):
            qs = rng.permutation(n)[:m].astype(np.int32)
            assert np.abs(sv.probs(qs) - o.probs(qs)).max() < 1e-14
            u = rng.uniform(size=(shots, m))
            assert np.array_equal(sv.sample(qs, u), o.sample(qs, u))
        assert abs(sv.prob_zero(n - 1) - o.probs([n - 1])[0]) < 1e-14


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n,m", [(3, 1), (9, 8), (9, 9), (10, 8), (10, 9), (11, 1), (11, 2), (11, 8), (11, 10)])
def test_threads_shared_among_few_bins(need_gpu, n, m, dtype):
    """Bins as wide as, narrower and wider than the CTA: several threads a bin, one, and several bins a thread."""
    rng = np.random.default_rng(50 * n + m)
    o = OracleState(n)
    o.apply(circuits.random_layers(n, 3, n))
    st = o.state()
    if dtype == "c64":
        st = st.astype(np.complex64).astype(np.complex128)
        o.set_state(st)
    with StateVector(n, dtype) as sv:
        sv.set_state(st.astype(np.complex64) if dtype == "c64" else st)
        for qs in (rng.permutation(n)[:m].astype(np.int32), np.arange(n - m, n, dtype=np.int32)):
            u = rng.uniform(size=(300, m))
            assert np.array_equal(sv.sample(qs, u), o.sample(qs, u))


def test_few_bins_take_no_longer_than_many(need_gpu):
    """One measured qubit of 11 is two bins of 1024 amplitudes: no more work than all 2048 bins."""
    rng = np.random.default_rng(0)

    def best(sv, qs):
        u = rng.uniform(size=(256, len(qs)))
        times = []
        for _ in range(40):
            t = time.perf_counter()
            sv.sample(qs, u)                  # waits for its result
            times.append(time.perf_counter() - t)
        return min(times)

    with StateVector(11, "c128") as sv:
        sv.apply(circuits.random_layers(11, 2, 1))
        assert best(sv, [4]) < 1.25 * best(sv, list(range(11)))
