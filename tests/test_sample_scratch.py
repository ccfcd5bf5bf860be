"""The sampler's scratch (CPU: the library's own layout).  The serving loop
admits a request with 64 MB of scratch, so a call of 1024 shots must fit that
with its buffer rounded up to a power of two, on every width and qubit list."""
import ctypes as C

import numpy as np
import pytest

from qpanda_b200.capi import lib

SERVED = 64 << 20


def scratch(n, dtype, qubits, shots=1024):
    f = lib().qs_sample_scratch_bytes
    f.restype = C.c_size_t
    f.argtypes = [C.c_int, C.c_int, C.POINTER(C.c_int), C.c_int, C.c_size_t]
    q = (C.c_int * len(qubits))(*qubits)
    need = f(n, dtype, q, len(qubits), shots)
    size = 1 << 20
    while size < need:
        size <<= 1
    return size


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("n", range(20, 33))
def test_all_qubits(n, dtype):
    # one slice: the tree of 20 levels (16 MB) and the shots
    assert scratch(n, dtype, range(n)) <= SERVED // 2
    assert scratch(n, dtype, range(n)[::-1]) <= SERVED // 2


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("n", [12, 16, 22, 27, 30, 32])
def test_any_qubits(n, dtype):
    rng = np.random.default_rng(n)
    for m in range(1, n + 1):
        for qubits in (list(range(m)), list(range(n - m, n)), [int(q) for q in rng.permutation(n)[:m]]):
            assert scratch(n, dtype, qubits) <= SERVED
