"""Downloads whose way depends on the arrays or on who else downloads: a batch
read by more threads than it keeps staging for, and state downloads into pages
that are untouched, touched or half and half.  Every value must arrive
exactly."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from code_mojo_gb300 import _ffi as F
from code_mojo_gb300 import butterfly as bfy
from code_mojo_gb300 import workloads as W
from code_mojo_gb300.batch import Batch

pytestmark = pytest.mark.gpu


# circuits on both sides of the directly copied size, 12 threads
@pytest.mark.parametrize("dtype", ["c128", "c64"])
def test_a_batch_read_by_many_threads(dtype):
    circuits = [W.random_layered_circuit(n, 2, n) for n in (2, 12, 13, 16, 17, 20)]
    b = Batch(circuits, dtype, tile_qubits=11)
    b.run()
    alone = [b.download(c) for c in range(len(circuits))]
    bad = []

    def read(start):
        for k in range(12):
            c = (start + k) % len(circuits)
            if not np.array_equal(b.download(c), alone[c]):
                bad.append(c)

    th = [threading.Thread(target=read, args=(k,)) for k in range(12)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    b.close()
    assert not bad


# 2^18 to 2^22 amplitudes: staged into untouched pages, copied by the driver
# into touched ones
@pytest.mark.parametrize("n", [17, 18, 20, 21])
def test_touched_and_untouched_arrays(n):
    N = 1 << n
    re, im = W.random_normal_state(n, n)
    st = bfy.QuantumState.from_soa(re, im)
    touched = [lambda: np.empty(N), lambda: np.ones(N), lambda: np.concatenate([np.ones(N // 2), np.empty(N // 2)]),
               lambda: np.empty(N + 1)[1:]]
    for a in touched:
        for b in touched:
            gr, gi = a(), b()
            F.check(F.lib().bf_state_download_soa(st.handle, gr.ctypes.data, gi.ctypes.data))
            assert np.array_equal(gr, re) and np.array_equal(gi, im)
    st.close()
