"""qs_plan_status reports on the last qs_plan_apply alone, also where a plan's
gates run one by one (below 12 qubits, complex128), and keeps its word when the
state's scratch grows between the two."""
import numpy as np
import pytest

from qpanda_b200 import FusionPlan, StateVector, circuits
from qpanda_b200.capi import QSError, check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dtype", [(11, "c64"), (12, "c64"), (12, "c128")])
def test_status_is_of_the_last_application(need_gpu, n, dtype):
    sv = StateVector(n, dtype)
    p = FusionPlan(n, circuits.random_layers(n, 2, n))
    check(lib().qs_watchdog_selftest(sv.handle, 50))
    u = np.random.default_rng(0).uniform(size=(200000, n))
    sv.sample(np.arange(n, dtype=np.int32), u)            # the scratch grows
    with pytest.raises(QSError):
        p.status(sv)                                      # and has not lost the word
    p.apply(sv)
    p.status(sv)
    p.close()
    sv.close()
