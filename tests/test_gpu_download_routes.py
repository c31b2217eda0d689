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
