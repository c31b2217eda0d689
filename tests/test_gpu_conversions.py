"""The FP64 <-> FP32-pair conversions of the double-float kernels, over the
whole exponent range: a phase of angle 0 multiplies an amplitude by exactly 1,
so what comes back is the value as a pair holds it.

Bounds: the pair keeps 47 significant bits above 2^-80 and its leading 24 (an
absolute 2^-103) below, nothing below 2^-126; values FP32's exponent cannot
hold become NaN; everything that leaves the pair is rounded once more to FP64."""
from __future__ import annotations

import numpy as np
import pytest

from code_mojo_gb300 import butterfly as bfy

pytestmark = pytest.mark.gpu


def values(n, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    m = rng.uniform(1, 2, 1 << n) * rng.choice([-1.0, 1.0], 1 << n)
    short = rng.integers(0, 53, 1 << n)  # few significant bits: powers of two and ties among them
    m = np.where(rng.random(1 << n) < 0.5, m, np.round(m * 2.0 ** short) / 2.0 ** short)
    e = rng.integers(-160, 128, 1 << n)
    e[: 1 << (n - 1)] = rng.integers(-40, 1, 1 << (n - 1))
    x = np.ldexp(m, e)
    x[:7] = [0.0, -0.0, 1.0, -1.0, 2.0 ** -126, 2.0 ** -80, np.nextafter(1.0, 0.0)]
    return x


@pytest.mark.parametrize("strategy,tile", [(bfy.ExecutionStrategy.GPU, 0), (bfy.ExecutionStrategy.GPU_FUSED, 9)])
def test_pairs_hold_their_bits(strategy, tile):
    n = 16
    re, im = values(n, 1), values(n, 2)
    qc = bfy.QuantumCircuit(n)
    for q in range(3 if tile else 1):  # (several, so that they make a tile pass)
        qc.custom(q, np.diag([1.0, 1.0]).astype(complex), [q + 3])
    for q in range(n):  # and one phase that touches every amplitude whose bit is 1
        qc.p(q, 0.0)
    ctx = bfy.ExecContext()
    ctx.execution_strategy = strategy
    ctx.gpu_tile_qubits = tile
    ctx.gpu_tensor_blocks = False
    st = bfy.QuantumState.from_soa(re, im)
    bfy.execute(st, qc, ctx)
    got = st.download()
    st.close()
    # (a component the pair cannot hold makes its partner NaN too)
    held = np.maximum(np.abs(re), np.abs(im)) < 2.0 ** 128
    for x, g in zip((re, im), got):
        a = np.abs(x)
        big = a >= 2.0 ** 127
        assert np.all(np.isnan(g[big & (a >= 2.0 ** 128)]))
        tiny = a < 2.0 ** -126
        assert np.all(np.abs(g[tiny & held]) <= a[tiny & held])
        mid = ~big & ~tiny & held
        bound = np.where(a >= 2.0 ** -80, a * 2.0 ** -46, 2.0 ** -100)  # a round trip per phase of its 16 bits at most
        assert np.all(np.abs(g - x)[mid] <= 8 * bound[mid])


def test_infinities_and_nans_stay_visible():
    re, im = np.zeros(16), np.zeros(16)
    re[1], re[3], im[5], re[7] = np.inf, -np.inf, np.nan, 1e300
    st = bfy.QuantumState.from_soa(re, im)
    qc = bfy.QuantumCircuit(4)
    qc.p(0, 0.0)
    ctx = bfy.ExecContext()
    ctx.execution_strategy = bfy.ExecutionStrategy.GPU
    bfy.execute(st, qc, ctx)
    gr, gi = st.download()
    st.close()
    assert not np.isfinite(gr[1]) and not np.isfinite(gr[3]) and np.isnan(gi[5]) and not np.isfinite(gr[7])
    assert np.all(gr[[0, 2, 4, 6]] == 0)
