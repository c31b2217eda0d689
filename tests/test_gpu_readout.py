"""Outcome probabilities read in contiguous tiles, and Grover loops applied as
one affine map, against numpy in 64 bits.

Tolerances: a probability is a sum of squares of total 1 accumulated with
about 46 significant bits, and a loop adds one FP64 offset to amplitudes of
norm 1 whose sum is good to 2^-46 of the state's 1-norm; both stay inside the
engine's parity bar of 1e-12 (complex128).  complex64 squares exact FP32
values, so its probabilities meet the same bar against the rounded state."""
from __future__ import annotations

import numpy as np
import pytest

from code_mojo_gb300 import butterfly as bfy
from code_mojo_gb300 import workloads as W
from tests.test_gpu_grover_loop import loop_body

pytestmark = pytest.mark.gpu
TOL = 1e-12


def expected(z, n, qubits, values):
    p = (z.real.astype(np.float64) ** 2 + z.imag.astype(np.float64) ** 2).reshape([2] * n)  # axis k = qubit n-1-k
    free = [q for k, q in enumerate(qubits) if values is None or values[k] is None]
    for k, q in enumerate(qubits):
        if values is not None and values[k] is not None:
            p = np.take(p, [int(values[k])], axis=n - 1 - q)
    gone = tuple(n - 1 - q for q in range(n) if q not in free)
    p = p.sum(axis=gone)  # axes: the free qubits, descending
    left = sorted(free, reverse=True)
    return p.transpose([left.index(q) for q in reversed(free)]).reshape(-1)  # first listed qubit fastest


# tile edge at 11 qubits; registers inside, above and across it; 0 to all
# qubits listed; ascending, descending and mixed order; fixed values on both sides
@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("n", [1, 4, 8, 10, 11, 12, 13, 17, 20])
def test_probabilities_of_any_register(n, dtype):
    re, im = W.random_normal_state(n, n)
    st = bfy.QuantumState.from_soa(re, im, dtype)
    z = re + 1j * im if dtype == "c128" else re.astype(np.float32) + 1j * im.astype(np.float32)
    rng = np.random.Generator(np.random.PCG64(n))
    every = list(range(n))
    lists = [[], every, every[::-1], [0], [n - 1], every[: n // 2], every[n // 2:]]
    lists += [[int(q) for q in rng.permutation(n)[:k]] for k in (1, max(1, n // 3), n)]
    for q in lists:
        values = [None] * len(q)
        assert np.max(np.abs(st.probabilities(q) - expected(z, n, q, None))) <= TOL
        for k in range(0, len(q), 3):
            values[k] = int(rng.integers(0, 2))
        assert np.max(np.abs(st.probabilities(q, values) - expected(z, n, q, values))) <= TOL
    st.close()


def iterate(z, marked, iters):
    for _ in range(iters):
        for m in marked:
            z[m] = -z[m]
        z = 2 * z.mean() - z
    return z


# one CTA (12 qubits) against several (13, 15); odd and even counts; no, one,
# eight and (at 3 qubits) every amplitude marked
@pytest.mark.parametrize("n,marked", [(3, list(range(8))), (3, []), (5, [31]), (12, [0, 4095]), (13, [8191]),
                                      (13, []), (15, [1, 2, 3, 500, 4096, 20000, 32766, 32767])])
@pytest.mark.parametrize("iters", [2, 3, 70, 1001])
def test_loop_is_the_repeated_iteration(n, marked, iters):
    re, im = W.random_normal_state(n, 3 * n + iters)
    st = bfy.QuantumState.from_soa(re, im)
    bfy.execute(st, loop_body(n, marked, iters))
    got = st.to_complex()
    st.close()
    assert np.max(np.abs(got - iterate(re + 1j * im, marked, iters))) <= TOL
