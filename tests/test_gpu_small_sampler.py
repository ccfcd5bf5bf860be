"""The one-CTA sampler of narrow states (up to 11 qubits) against the oracle's
literal per-shot re-measurement, and small marginals that land in the state's
pinned host buffer: widths on both sides of the limits, subsets in any order,
shots on both sides of the buffer's size."""
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
