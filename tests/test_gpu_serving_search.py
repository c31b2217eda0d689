"""Grover iterations of server requests (one affine map, as a sum and an update
launched apart): 1, 2 and many chunks, odd and even counts, several marked
indices, from a state that is not uniform, against the iterations one by one in
64 bits."""
from __future__ import annotations

import numpy as np
import pytest

from code_mojo_gb300 import butterfly as bfy
from code_mojo_gb300 import opsarray as OA
from code_mojo_gb300 import workloads as W
from code_mojo_gb300.serving import Server
from oracle import pyoracle as O
from tests.test_gpu_grover_loop import loop_body
from tests.test_gpu_readout import iterate

pytestmark = pytest.mark.gpu


def request(n, marked, iters):
    first = W.random_layered_circuit(n, 1, n)
    body = loop_body(n, marked, iters)
    arr, count, keep = first.to_ops()
    head = np.frombuffer(arr, dtype=OA.BF_OP, count=count)
    return first, OA.OpArray(n, np.concatenate([head, body.ops]), [arr, keep, body])


# chunks hold at least 2^12 amplitudes
@pytest.mark.parametrize("dtype,tol", [("c128", 1e-12), ("c64", 1e-6)])
def test_served_iterations(dtype, tol):
    asked, srv = {}, Server(slots=6)
    for n, marked in [(5, [3, 17]), (12, [4095]), (13, [0, 8191]), (14, []), (18, [7, 70000, 262143]), (21, [2 ** 20])]:
        for iters in (2, 3, 40):
            first, ops = request(n, marked, iters)
            asked[srv.submit(ops, dtype)] = (n, first, marked, iters, ops)
    assert srv.wait_idle(120.0)
    done = {r.id: r for r in srv.poll()}
    srv.close()
    for rid, (n, first, marked, iters, _) in asked.items():
        re, im = O.run(first, *O.basis(n))
        p = np.abs(iterate(re + 1j * im, marked, iters)) ** 2
        r = done[rid]
        assert r.status == 0
        assert np.max(np.abs(np.sort(p)[::-1][:len(r.top_prob)] - r.top_prob)) <= tol
        assert np.max(np.abs(p[r.top_index] - r.top_prob)) <= tol
