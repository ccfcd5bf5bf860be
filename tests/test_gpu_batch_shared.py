"""Batches whose widest circuits are shared among CTAs (qs_batch.cu): one
circuit alone at the smallest and at larger widths, a wide one beside many
narrow ones, circuits of unequal depth in step.  <Z_i Z_{i+1}> against the
FP64 oracle within the batch tests' tolerance (a complex64 state after fused
tensor-core passes), states and replays of the graph with it."""
import numpy as np
import pytest

from qpanda_b200 import Batch, circuits
from tests.test_gpu_batch import TOL, oracle_zz

pytestmark = pytest.mark.gpu

SWEEPS = {
    "alone_14": [(14, 3)],
    "alone_18": [(18, 4)],
    "wide_beside_narrow": [(19, 3)] + [(8 + k % 6, 1 + k % 4) for k in range(40)],
    "unequal": [(17, 1), (16, 5), (18, 2), (14, 4), (17, 4)],
}


@pytest.mark.parametrize("name", list(SWEEPS))
@pytest.mark.parametrize("order", [0, 1])
def test_shared_circuits_match_oracle(need_gpu, name, order):
    sweep = [(q, circuits.vqe_ansatz(q, layers, seed=100 * q + layers)) for q, layers in SWEEPS[name]]
    b = Batch(sweep, order=order)
    b.run()
    zz = b.zz()
    for _ in range(3):                       # the same bits every time, whichever CTA takes which part
        b.run()
        assert all(np.array_equal(a, c) for a, c in zip(zz, b.zz()))
    for k, (q, g) in enumerate(sweep):
        ref_zz, ref_state = oracle_zz(q, g)
        assert np.abs(zz[k] - ref_zz).max() < TOL, (k, q)
        assert np.abs(b.state(k) - ref_state).max() < TOL, (k, q)


@pytest.mark.parametrize("count,width", [(296, 13), (297, 13), (64, 12), (888, 16)])
def test_lane_groups_match_oracle(need_gpu, count, width):
    """Both sides of the rule for lane groups per CTA: circuits of one, two and
    16 tiles, up to and past one circuit per CTA, one odd width among them."""
    few = [(width, circuits.vqe_ansatz(width, 1 + k, seed=7 * width + k)) for k in range(2)]
    few.append((width + 1, circuits.vqe_ansatz(width + 1, 2, seed=5)))
    refs = [oracle_zz(q, g)[0] for q, g in few]
    b = Batch([few[k % 2] for k in range(count - 1)] + [few[2]])
    b.run()
    zz = b.zz()
    for k in range(count):
        assert np.abs(zz[k] - refs[2 if k == count - 1 else k % 2]).max() < TOL, k


def test_non_finite_angle_reaches_every_amplitude(need_gpu):
    """Zero times NaN is no zero: tiles that the passes would leave alone take
    part when a circuit of their structure has an angle that is not finite, as
    they do in the kernel that leaves none alone.  The highest qubits are idle."""
    def circuit(n, theta):
        return n, circuits.make_gates([("RX", (0,), theta)] + [("RY", (q,), 0.3 + q) for q in range(1, 11)])

    sweep = [circuit(14, np.nan), circuit(14, 0.7), circuit(17, np.nan)]
    states = {}
    for tmem in (0, 1):
        b = Batch(sweep, tile_in_tmem=tmem)
        b.run()
        assert np.isnan(b.zz()[0]).all() and np.isnan(b.zz()[2]).all()
        states[tmem] = [b.state(k) for k in range(3)]
    for k in range(3):
        assert np.array_equal(np.isnan(states[1][k]), np.isnan(states[0][k])), k
    assert np.isnan(states[1][0]).all() and np.isnan(states[1][2]).all()
    assert np.abs(states[1][1] - oracle_zz(*sweep[1])[1]).max() < TOL
