"""The half sums of qs_prob_zero, qs_measure and qs_norm2 (one launch; the CTA
that ends last adds the partials): one CTA and many, repeated on one state and
on two states in turn, against numpy's FP64 sums.  Tolerance: a sum of 2^n
squares in FP64, 2^n * 2^-53 relative at the very worst; inputs to 2^18."""
import numpy as np
import pytest

from qpanda_b200 import StateVector
from qpanda_b200.capi import QSError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n", [1, 2, 9, 10, 11, 18])
def test_half_sums(need_gpu, n, dtype):
    rng = np.random.default_rng(n)
    svs, refs = [], []
    for _ in range(2):
        a = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
        a = (a / np.linalg.norm(a)).astype(np.complex64 if dtype == "c64" else np.complex128)
        sv = StateVector(n, dtype)
        sv.set_state(a)
        svs.append(sv)
        refs.append(np.abs(a.astype(np.complex128)) ** 2)
    tol = 2.0 ** (n - 53)
    for q in range(n):
        for sv, p in zip(svs, refs):
            zero = p.reshape(-1, 2, 1 << q)[:, 0].sum()
            assert abs(sv.prob_zero(q) - zero) <= tol + 4e-16
            assert abs(sv.norm2() - p.sum()) <= tol + 4e-16
    for sv, p in zip(svs, refs):
        q = n - 1
        zero = p.reshape(-1, 2, 1 << q)[:, 0].sum()
        u = 0.5 * (1 + zero)
        assert sv.measure(q, u) == 1                      # u above P(0)
        got = sv.get_state().reshape(-1, 2, 1 << q)
        assert not got[:, 0].any()
        eps = 1.2e-7 if dtype == "c64" else 2.3e-16       # rounding of the scale and of the product
        assert abs((np.abs(got) ** 2).sum() - p.sum() / (1 - zero) + zero / (1 - zero)) <= 8 * eps
        with pytest.raises(QSError):                      # 0 > P(0) = 0 fails: outcome 0, of probability 0
            sv.measure(q, 0.0)
        sv.close()
