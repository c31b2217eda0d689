"""<a|b> of states of either dtype at the sizes where its loop changes: one
load per thread, four in flight (from 2^20 amplitudes on, with 8 CTAs of 256
threads per SM) and the remainder between, against numpy in 64 bits.

Bound: each product and sum keeps about 46 bits of terms whose magnitudes sum
to at most 1 (unit norms)."""
from __future__ import annotations

import numpy as np
import pytest

from code_mojo_gb300 import butterfly as bfy
from code_mojo_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("da,db", [("c128", "c128"), ("c128", "c64"), ("c64", "c128"), ("c64", "c64")])
@pytest.mark.parametrize("n", [1, 7, 12, 18, 19, 20, 21, 22])
def test_inner_product(n, da, db):
    za, zb = [], []
    states = []
    for seed, dt in ((1, da), (2, db)):
        re, im = W.random_normal_state(n, seed + n)
        if dt == "c64":
            re, im = (x.astype(np.float32).astype(np.float64) for x in (re, im))
        states.append(bfy.QuantumState.from_soa(re, im, dt))
        (za if seed == 1 else zb).append(re + 1j * im)
    got = states[0].inner(states[1])
    for s in states:
        s.close()
    assert abs(got - np.vdot(za[0], zb[0])) <= 2.0 ** -42
