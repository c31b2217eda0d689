"""Phase gates merged into fans: the merged passes, applied on the host from
their tables (tests/fan_model.cpp), and on the GPU, against the oracle's gate
by gate run.

Tolerances: the host model multiplies unit phases in FP64, a few hundred
roundings of 2^-53 on amplitudes below 1 (1e-13); on the GPU the engine's
parity bars (1e-12 at complex128, 1e-6 infidelity at complex64)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from code_mojo_gb300 import butterfly as bfy
from code_mojo_gb300 import workloads as W
from code_mojo_gb300.batch import Batch
from oracle import pyoracle as O

ROOT = Path(__file__).resolve().parent.parent
CUDA_INC = Path("/usr/local/cuda/include")


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    if shutil.which("g++") is None or not CUDA_INC.exists():
        pytest.skip("needs g++ and the CUDA headers")
    from code_mojo_gb300 import build
    lib = build.build_engine()
    exe = tmp_path_factory.mktemp("fan_model") / "fan_model"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(CUDA_INC), "-I", str(ROOT / "include"),
                    str(ROOT / "tests" / "fan_model.cpp"), "-o", str(exe), "-L", str(lib.parent), "-lbfgpu",
                    f"-Wl,-rpath,{lib.parent}"], check=True, capture_output=True)
    return exe


def phase_mix(n, count, seed, diag=True):
    """Phases of one to four qubits in any order among gates of every other
    kind, controls and targets anywhere."""
    rng = np.random.Generator(np.random.PCG64(seed))
    qc = bfy.QuantumCircuit(n)
    for _ in range(count):
        q = [int(x) for x in rng.permutation(n)[:4]]
        a = float(rng.uniform(0, 2 * np.pi))
        k = int(rng.integers(0, 12 if diag else 11))
        if k <= 1 or n < 4 and k <= 5:
            qc.p(q[0], a)
        elif k <= 4:
            qc.cp(q[0], q[1], a)
        elif k == 5:
            qc.mcp(q[:2 + int(rng.integers(0, 2))], q[3], a)
        elif k == 6:
            qc.h(q[0])
        elif k == 7:
            qc.u3(q[0], a, 0.3, -a)
        elif k == 8:
            qc.ry(q[0], a)
        elif k == 9 and n > 1:
            qc.cx(q[0], q[1])
        elif k == 10 and n > 1:
            qc.cry(q[0], q[1], a)
        elif k == 11:
            qc.rz(q[0], a)
        else:
            qc.x(q[0])
    return qc


def gates_only(qc):
    out = bfy.QuantumCircuit(qc.num_qubits)
    out.transformations = [t for t in qc.transformations if isinstance(t, bfy.GateTransformation)]
    return out


def with_unitaries(n, seed):
    qc = phase_mix(n, 60, seed)
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    for m in (2, 3, 5):
        u = np.linalg.qr(rng.standard_normal((1 << m, 1 << m)) + 1j * rng.standard_normal((1 << m, 1 << m)))[0]
        qc.unitary(u, int(rng.integers(0, n - m + 1)), m)
        qc.transformations += phase_mix(n, 25, seed + m).transformations
    return qc


CIRCUITS = {
    "qft": lambda n: gates_only(W.qft_circuit(n)),
    "encode": lambda n: W.encode_value_circuit(n, 3.7),
    "encode_lsb": lambda n: W.value_encoding_phase_circuit(n, 5.3),
    "phases_only": lambda n: phase_mix_phases(n),
    "mix1": lambda n: phase_mix(n, 120, 1),
    "mix2": lambda n: phase_mix(n, 200, 2, diag=False),
}


def phase_mix_phases(n):
    qc = bfy.QuantumCircuit(n)
    for i in range(n):
        for j in range(i):
            qc.cp(j, i, 0.1 * (i + 1) / (j + 1))
    return qc


def run_model(exe, qc, re, im, K, units, tmp_path):
    ops, sin, sout = tmp_path / "ops.bin", tmp_path / "in.bin", tmp_path / "out.bin"
    ops.write_bytes(bfy.serialize(qc))
    (re + 1j * im).astype(np.complex128).tofile(sin)
    r = subprocess.run([str(exe), str(ops), str(sin), str(sout), str(K), str(units)], check=True, capture_output=True,
                       text=True)
    return np.fromfile(sout, dtype=np.complex128), [int(x) for x in r.stdout.split()]


# tiles from 1 qubit to the whole state, odd widths among them; plans with and
# without tensor-core blocks in view
@pytest.mark.parametrize("name", list(CIRCUITS))
@pytest.mark.parametrize("n,K,units", [(3, 11, 0), (7, 1, 0), (7, 6, 0), (10, 7, 0), (11, 11, 0), (13, 12, 2.5), (14, 12, 3.3),
                                       (13, 9, 0), (14, 13, 0)])
def test_merged_passes_match_the_oracle(model, name, n, K, units, tmp_path):
    qc = CIRCUITS[name](n)
    re, im = W.random_normal_state(n, 11)
    got, _ = run_model(model, qc, re, im, K, units, tmp_path)
    r, i = O.run(qc, re, im)
    assert np.max(np.abs(got - (r + 1j * i))) <= 1e-13


def test_merged_passes_with_unitaries(model, tmp_path):
    for n, K in ((9, 9), (13, 11), (13, 12)):
        qc = with_unitaries(n, n)
        re, im = W.random_normal_state(n, 12)
        got, _ = run_model(model, qc, re, im, K, 0, tmp_path)
        r, i = O.run(qc, re, im)
        assert np.max(np.abs(got - (r + 1j * i))) <= 1e-13


def test_a_qft_keeps_one_fan_per_hadamard(model, tmp_path):
    """Every phase joins the fan before the gate that meets it: at most one
    fan per Hadamard, and only a Hadamard's lone phase is left as an op."""
    n = 14
    qc = CIRCUITS["qft"](n)
    re, im = W.random_normal_state(n, 13)
    _, (tiles, _, fans, phases) = run_model(model, qc, re, im, 11, 0, tmp_path)
    assert tiles <= 2 and fans <= n and phases <= 1


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("name", list(CIRCUITS) + ["unitaries"])
@pytest.mark.parametrize("n,K", [(3, 0), (8, 8), (9, 0), (11, 0), (12, 12), (15, 7), (15, 11), (16, 12), (16, 13)])
def test_fans_on_the_gpu(name, n, K, dtype):
    if name == "unitaries" and n < 8:
        pytest.skip("needs five contiguous qubits beside the phases")
    qc = with_unitaries(n, n) if name == "unitaries" else CIRCUITS[name](n)
    re, im = W.random_normal_state(n, 21)
    ctx = bfy.ExecContext()
    ctx.gpu_tile_qubits = K
    ctx.gpu_tensor_blocks = K == 0
    st = bfy.QuantumState.from_soa(re, im, dtype)
    bfy.execute(st, qc, ctx)
    got = st.to_complex()
    st.close()
    r, i = O.run(qc, re, im)
    exp = r + 1j * i
    if dtype == "c128":
        assert np.max(np.abs(got - exp)) <= 1e-12
    else:
        assert 1 - abs(np.vdot(exp, got)) ** 2 / (np.vdot(exp, exp).real * np.vdot(got, got).real) <= 1e-6


@pytest.mark.gpu
def test_fans_in_fp64_arithmetic(monkeypatch):
    monkeypatch.setenv("BFGPU_C128_MATH", "f64")
    test_fans_on_the_gpu("mix1", 15, 11, "c128")
    test_fans_on_the_gpu("encode", 16, 12, "c128")


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("width", [0, 5, 9])
def test_fans_in_a_batch(dtype, width):
    """Circuits with and without fans in one launch."""
    circuits = [CIRCUITS[k](n) for k in ("encode", "mix1", "qft") for n in (3, 9, 12, 14)]
    circuits += [W.random_layered_circuit(n, 3, n) for n in (5, 13)]
    b = Batch(circuits, dtype, tile_qubits=width)
    b.run()
    for c, qc in enumerate(circuits):
        r, i = O.run(qc, *O.basis(qc.num_qubits))
        exp, got = r + 1j * i, b.download(c)
        if dtype == "c128":
            assert np.max(np.abs(got - exp)) <= 1e-12
        else:
            assert 1 - abs(np.vdot(exp, got)) ** 2 / (np.vdot(exp, exp).real * np.vdot(got, got).real) <= 1e-6
    b.close()
