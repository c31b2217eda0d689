"""Downloads into ordinary host arrays at the sizes where their way changes
(2^14, 2^18 and 2^22 amplitudes), ranges that start anywhere, and a batch's
circuits read by several threads at once.  Every value must arrive exactly
(complex64 states hold the FP32 rounding of the input)."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from code_mojo_gb300 import _ffi as F
from code_mojo_gb300 import butterfly as bfy
from code_mojo_gb300 import workloads as W
from code_mojo_gb300.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("n", [1, 13, 14, 17, 18, 20, 21])
def test_round_trip_is_exact(n, dtype):
    rng = np.random.Generator(np.random.PCG64(n))
    re, im = rng.standard_normal(1 << n), rng.standard_normal(1 << n)
    st = bfy.QuantumState.from_soa(re, im, dtype)
    if dtype == "c64":
        re, im = re.astype(np.float32).astype(np.float64), im.astype(np.float32).astype(np.float64)
    for _ in range(2):  # the second one reuses the staging
        gr, gi = st.download()
        assert np.array_equal(gr, re) and np.array_equal(gi, im)
    N = 1 << n
    for off, cnt in [(0, N), (N // 3, min(N - N // 3, (1 << 14) - 1)), (N // 2, N - N // 2), (N - 1, 1),
                     (0, min(N, (1 << 18) + 5)), (N // 5, 0)]:
        gr, gi = np.empty(cnt), np.empty(cnt)
        F.check(F.lib().bf_state_download_range(st.handle, off, cnt, gr.ctypes.data, gi.ctypes.data))
        assert np.array_equal(gr, re[off:off + cnt]) and np.array_equal(gi, im[off:off + cnt])
    st.close()


def test_batch_downloads_from_several_threads():
    circuits = [W.random_layered_circuit(n, 2, n) for n in (3, 14, 15, 18, 20)]
    b = Batch(circuits, "c128", tile_qubits=11)
    b.run()
    alone = [b.download(c) for c in range(len(circuits))]
    bad = []

    def read(start):
        for k in range(10):
            c = (start + k) % len(circuits)
            if not np.array_equal(b.download(c), alone[c]):
                bad.append(c)

    th = [threading.Thread(target=read, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    b.close()
    assert not bad
