"""The digit kernel's choice of five or six digits where a warp's quick sum of
squares does not decide: the counts follow the exact per-value bound, and the
two forms give the same bits."""
from __future__ import annotations

import numpy as np
import pytest

from code_mojo_gb300 import butterfly as bfy

CAP = 1 << 27


def exact_units(x: float, e: int) -> int:
    """x^2 in units of 2^(2e - 50), rounded up as (257 + top 8 mantissa bits)^2 2^k."""
    m, ex = np.frexp(x)  # x = m 2^ex, 1/2 <= m < 1
    u = 257 + (int(m * 512) - 256)
    k = 2 * (int(ex) - 9 - e) + 50
    return min(u * u << k, CAP) if k >= 0 else -(-(u * u) >> -k)


@pytest.mark.gpu
@pytest.mark.parametrize("n,qubits", [(13, 5), (14, 14)])
@pytest.mark.parametrize("r", [0.95, 0.986, 0.99, 0.994, 0.998, 1.002, 1.005, 1.05])
def test_tiles_near_the_norm_bound(monkeypatch, r, n, qubits):
    """Every component is c, 256 c^2 = r 2^27 units at scale 2^9: about the
    limit of a warp.  X and Y turn no magnitude, so later passes, which read
    integers, meet the same sums as the first, which reads FP64."""
    c = np.sqrt(r * 2.0 ** -13)
    re, im = np.full(1 << n, c), np.full(1 << n, c)
    qc = bfy.QuantumCircuit(n)
    for q in range(qubits):
        qc.x(q)
        qc.y(q)
    ctx = bfy.ExecContext()
    ctx.execution_strategy = bfy.ExecutionStrategy.GPU_FUSED
    plan = bfy.plan_stats(qc, ctx, "c128")
    passes = plan["block_passes"]
    assert passes == plan["tile_passes"] == (1 if qubits == 5 else 2) and plan["gate_kernels"] == 0
    norm = np.sqrt(np.sum(re * re) + np.sum(im * im))
    shift = 9 - (int(np.frexp(norm * (1.0 + 1e-6))[1]) + 1)
    six = 256 * exact_units(c, 9) >= CAP
    tiles = passes << (n - 12)
    monkeypatch.setenv("BFGPU_DIGIT_SCALE_SHIFT", str(shift))
    out = []
    for five in ("1", "0"):
        monkeypatch.setenv("BFGPU_DIGIT_FIVE", five)
        st = bfy.QuantumState.from_soa(re, im, "c128")
        st.digit_tiles(reset=True)
        bfy.execute(st, qc, ctx)
        got = st.digit_tiles()
        if five == "1":
            assert got == ((0, tiles) if six else (tiles, 0))
        else:
            assert got == (0, tiles)
        out.append(st.to_complex())
        st.close()
    assert np.array_equal(out[0], out[1])
