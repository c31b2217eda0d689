"""Outcome probabilities with fixed qubits among the low index bits, where a
tile of the readout is not contiguous, and registers whose outcomes are summed
over many chunks, against numpy in 64 bits (the tolerance of
test_gpu_readout)."""
from __future__ import annotations

import numpy as np
import pytest

from code_mojo_gb300 import butterfly as bfy
from code_mojo_gb300 import workloads as W
from tests.test_gpu_readout import TOL, expected

pytestmark = pytest.mark.gpu


def check(st, z, n, fixed, free, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    q = [int(x) for x in rng.permutation(fixed + free)]
    values = [int(rng.integers(0, 2)) if x in fixed else None for x in q]
    assert np.max(np.abs(st.probabilities(q, values) - expected(z, n, q, values))) <= TOL


# the unfixed qubits fill less than a warp, less than a tile, a tile exactly
# (11), and one qubit more
@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("n", [6, 11, 12, 15, 18])
def test_fixed_low_qubits(n, dtype):
    re, im = W.random_normal_state(n, n)
    st = bfy.QuantumState.from_soa(re, im, dtype)
    z = re + 1j * im if dtype == "c128" else re.astype(np.float32) + 1j * im.astype(np.float32)
    for left in (0, 1, 5, 8, 10, 11, 12):
        if left > n:
            continue
        low, high = list(range(n - left)), list(range(n - left, n))
        for free in ([], high[:1], high[-1:], high[::2], high):
            check(st, z, n, low, free, 7 * n + left)
    for fixed in ([0], [5], [10], [0, 1, 2], list(range(0, n, 2)), list(range(1, n, 3)), [n - 1, 0]):
        fixed = sorted({q for q in fixed if q < n})
        rest = [q for q in range(n) if q not in fixed]
        for free in ([], rest[:3], rest[-2:], rest[::3], rest):
            check(st, z, n, fixed, free, n + len(fixed))
    st.close()


# the sums of 1 to 1024 chunks, of registers narrower and wider than the
# chunk kernel's rows
@pytest.mark.parametrize("n", [14, 19, 22])
def test_chunk_sums(n):
    re, im = W.random_normal_state(n, n)
    st = bfy.QuantumState.from_soa(re, im)
    z = re + 1j * im
    for k in (0, 1, 2, 5, 6, 9):
        check(st, z, n, [], list(range(k)), k)
        check(st, z, n, [], list(range(n - k, n)), k)
    st.close()
