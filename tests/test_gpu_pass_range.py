"""Hadamards of a tile pass run in pairs without their factors: the pass must
give every amplitude its right power of two, and stay inside FP32's exponent
range wherever the gates one by one do.  Amplitudes are compared directly, with
no norm restored and none divided out.

Bound: a gate or phase rounds each amplitude of a pair to a few units of the
arithmetic (2^-24 at complex64, 2^-45 for a double-float product), so a circuit
of G ops is off by at most 4 G units of the state's norm."""
from __future__ import annotations

import numpy as np
import pytest

from code_mojo_gb300 import butterfly as bfy
from code_mojo_gb300 import workloads as W
from code_mojo_gb300.batch import Batch
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def hadamards(n, times):
    qc = bfy.QuantumCircuit(n)
    for _ in range(times):
        for q in range(n):
            qc.h(q)
    return qc


def qft_gates(n):
    out = bfy.QuantumCircuit(n)
    out.transformations = [t for t in W.qft_circuit(n).transformations if isinstance(t, bfy.GateTransformation)]
    return out


CIRCUITS = {
    "h": lambda n: hadamards(n, 1),          # an odd number of factors at odd n
    "hh": lambda n: hadamards(n, 2),
    "hhh": lambda n: hadamards(n, 3),
    "qft": qft_gates,
    "encode": lambda n: W.encode_value_circuit(n, 2.7),
}


def off(got, exp):
    return np.linalg.norm(got - exp) / np.linalg.norm(exp)


# 2^120: a pass of 12 pairs has no room for its factors' 2^12
@pytest.mark.parametrize("scale", [0, 120, -60])
@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("name", list(CIRCUITS))
@pytest.mark.parametrize("n,K", [(1, 0), (5, 5), (7, 0), (12, 12), (13, 9)])
def test_amplitudes_keep_their_scale(name, n, K, dtype, scale):
    qc = CIRCUITS[name](n)
    re, im = W.random_normal_state(n, 31)
    if dtype == "c64":
        re, im = (x.astype(np.float32).astype(np.float64) for x in (re, im))
    ctx = bfy.ExecContext()
    ctx.gpu_tile_qubits = K
    ctx.gpu_tensor_blocks = False
    ctx.gpu_renormalize = False
    st = bfy.QuantumState.from_soa(np.ldexp(re, scale), np.ldexp(im, scale), dtype)
    bfy.execute(st, qc, ctx)
    gr, gi = st.download()
    st.close()
    r, i = O.run(qc, re, im)
    unit = 2.0 ** -24 if dtype == "c64" else 2.0 ** -45
    assert off(np.ldexp(gr, -scale) + 1j * np.ldexp(gi, -scale), r + 1j * i) <= 4 * len(qc.transformations) * unit


@pytest.mark.parametrize("dtype", ["c128", "c64"])
def test_a_batch_keeps_the_factors(dtype):
    names = [(k, n) for k in CIRCUITS for n in (1, 6, 11, 13)]
    b = Batch([CIRCUITS[k](n) for k, n in names], dtype, tile_qubits=9)
    b.run()
    for c, (k, n) in enumerate(names):
        qc = CIRCUITS[k](n)
        r, i = O.run(qc, *O.basis(n))
        unit = 2.0 ** -24 if dtype == "c64" else 2.0 ** -45
        assert off(b.download(c), r + 1j * i) <= 4 * len(qc.transformations) * unit
    b.close()


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("inside", [True, False])
def test_factors_that_are_no_phases(dtype, inside):
    """diag(1, 2^60) and diag(1, 2^-60) in turn: every amplitude of the state
    goes up and comes back, though the product of either kind overflows.  The
    factors are powers of two, so the amplitudes return exactly."""
    n = 9
    qc = bfy.QuantumCircuit(n)
    up, down = ((1, 2, 3), (5, 6, 7)) if inside else ((8, 7, 6), (1, 2, 3))
    for a, b in zip(up, down):
        qc.custom(0, np.diag([1.0, 2.0 ** 60]).astype(complex), [a])
        qc.custom(0, np.diag([1.0, 2.0 ** -60]).astype(complex), [b])
    x = np.arange(1 << n)
    paired = np.all([(x >> a & 1) == (x >> b & 1) for a, b in zip(up, down)], axis=0)
    re, im = (np.where(paired, v.astype(np.float32), 0.0).astype(np.float64) for v in W.random_normal_state(n, 41))
    ctx = bfy.ExecContext()
    ctx.gpu_tile_qubits = 8 if inside else 6
    ctx.gpu_tensor_blocks = False
    ctx.gpu_renormalize = False
    st = bfy.QuantumState.from_soa(re, im, dtype)
    bfy.execute(st, qc, ctx)
    gr, gi = st.download()
    st.close()
    assert np.array_equal(gr, re) and np.array_equal(gi, im)


@pytest.mark.parametrize("n", [9, 12, 15, 18, 20])
def test_complex64_value_encoding_stays_near_fp32(n):
    """About three roundings of half a unit per Hadamard and its fan along the
    way of an amplitude, 2 n of them: as a random walk sqrt(6 n) units of 2^-24
    at three standard deviations, and one for the stored value; in the largest
    amplitude and in the norm of the error alike."""
    bound = (np.sqrt(6 * n) + 1) * 2.0 ** -24
    for v in (0.37, 2 ** (n - 1) + 0.5, 2 ** n - 1.21):
        qc = W.encode_value_circuit(n, v)
        st = bfy.QuantumState(n, "c64")
        bfy.execute(st, qc)
        got = st.to_complex()
        st.close()
        r, i = O.run(qc, *O.basis(n))
        d = got - (r + 1j * i)
        assert np.max(np.abs(d)) <= bound and np.linalg.norm(d) <= bound


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("times", [2, 24])
def test_factors_over_the_exponent_range(dtype, times):
    """H an even number of times on one qubit, 1 and 12 powers of two at the
    store, on amplitudes from below the smallest values a pair keeps whole up
    to where a pass scales its tiles before the gates (2^100) and beyond.

    Each H rounds by a few units of the larger amplitude of the pair; below,
    an absolute 2^-100 (what a pair drops, with the tile scaled by 2^-12)."""
    n = 14
    rng = np.random.Generator(np.random.PCG64(times))
    e = rng.integers(-140, 100, 1 << n)
    e[1 << 9:3 << 9] = rng.integers(-40, 125, 2 << 9)   # tiles with large amplitudes beside tiles without
    e[5 << 9:6 << 9] = rng.integers(98, 102, 1 << 9)
    x = np.ldexp(rng.uniform(1, 2, (2, 1 << n)) * rng.choice([-1.0, 1.0], (2, 1 << n)), e)
    if dtype == "c64":
        x = x.astype(np.float32).astype(np.float64)
    qc = bfy.QuantumCircuit(n)
    for _ in range(times):
        qc.h(3)
    ctx = bfy.ExecContext()
    ctx.gpu_tile_qubits = 9
    ctx.gpu_tensor_blocks = False
    ctx.gpu_renormalize = False
    st = bfy.QuantumState.from_soa(x[0], x[1], dtype)
    bfy.execute(st, qc, ctx)
    got = np.array(st.download())
    st.close()
    pair = np.abs(x).max(0).reshape(-1, 2, 8)           # qubit 3
    top = np.broadcast_to(pair.max(1, keepdims=True), pair.shape).reshape(-1)
    unit = 2.0 ** -24 if dtype == "c64" else 2.0 ** -45
    assert np.all(np.abs(got - x).max(0) <= 4 * times * unit * top + 2.0 ** -100)


@pytest.mark.parametrize("n,K", [(14, 5), (13, 4)])
def test_complex64_constants_round_once(n, K):
    """A phase on every set of the qubits outside the tile and one inside, then
    a Hadamard there: the constant of the fan is a product of up to 2^(n-K)
    factors and has to come out as one rounded number.

    Bound by pairs, in units of 2^-24 of a pair's norm: 1 for the constant,
    sqrt(5) for a complex product, 3 for the Hadamard (sum, factor, product);
    a constant whose products are rounded one by one is off by about 14."""
    rng = np.random.Generator(np.random.PCG64(n))
    qc = bfy.QuantumCircuit(n)
    for m in range(1, 1 << (n - K)):
        qc.mcp([K + j for j in range(n - K) if m >> j & 1], 2, float(rng.uniform(-3, 3)))
    qc.h(2)
    re, im = (x.astype(np.float32).astype(np.float64) for x in W.random_normal_state(n, 5))
    ctx = bfy.ExecContext()
    ctx.gpu_tile_qubits = K
    ctx.gpu_tensor_blocks = False
    ctx.gpu_renormalize = False
    st = bfy.QuantumState.from_soa(re, im, "c64")
    bfy.execute(st, qc, ctx)
    gr, gi = st.download()
    st.close()
    r, i = O.run(qc, re, im)
    pairs = lambda x: np.sqrt((np.abs(x).reshape(-1, 2, 4) ** 2).sum(1))
    err = pairs((gr - r) + 1j * (gi - i)) / pairs(r + 1j * i)
    assert np.max(err) <= (1 + np.sqrt(5) + 3) * 2.0 ** -24
