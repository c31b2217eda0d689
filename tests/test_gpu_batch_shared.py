"""One op list given for several circuits of a batch, in one call, among others
and at two sizes: each circuit has a state of its own, whatever its plan is
shared with."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from code_mojo_gb300 import _ffi as F
from code_mojo_gb300 import butterfly as bfy
from code_mojo_gb300 import workloads as W
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [F.BF_C128, F.BF_C64])
@pytest.mark.parametrize("width", [0, 6, 11])
def test_circuits_with_one_op_list(dtype, width):
    enc = W.encode_value_circuit(9, 3.3)                 # fans
    lay = W.random_layered_circuit(12, 3, 1)             # several passes
    qft = bfy.QuantumCircuit(9)
    qft.transformations = [t for t in W.qft_circuit(9).transformations if isinstance(t, bfy.GateTransformation)]
    lists = [c.to_ops() for c in (enc, lay, qft)]
    # (list, qubits): the value encoding also on the low 9 of 13 qubits
    plan = [(0, 9), (1, 12), (0, 9), (2, 9), (0, 13), (1, 12), (0, 13), (2, 9), (0, 9), (1, 14)]
    opts = F.bf_exec_opts()
    F.check(F.lib().bf_exec_opts_init(C.byref(opts)))
    opts.tile_qubits = width
    k = len(plan)
    nq = (C.c_int32 * k)(*[n for _, n in plan])
    nops = (C.c_int64 * k)(*[lists[i][1] for i, _ in plan])
    ptrs = (C.c_void_p * k)(*[C.addressof(lists[i][0]) for i, _ in plan])
    h = C.c_void_p()
    F.check(F.lib().bf_batch_create(k, nq, ptrs, nops, dtype, C.byref(opts), C.byref(h)))
    try:
        for _ in range(2):
            F.check(F.lib().bf_batch_run(h, 1))
            for c, (i, n) in enumerate(plan):
                re, im = np.empty(1 << n), np.empty(1 << n)
                F.check(F.lib().bf_batch_download(h, c, re.ctypes.data, im.ctypes.data))
                qc = bfy.QuantumCircuit(n)
                qc.transformations = (enc, lay, qft)[i].transformations
                r, m = O.run(qc, *O.basis(n))
                unit = 2.0 ** -46 if dtype == F.BF_C128 else 2.0 ** -24
                d = np.linalg.norm((re - r) + 1j * (im - m))
                assert d <= 4 * len(qc.transformations) * unit, (c, i, n, d)
    finally:
        F.check(F.lib().bf_batch_destroy(h))
