"""Planning circuits of many phases: the phases that wait in a pass are one per
mask and found by the qubits that a gate acts on, so that planning time grows
with the gate count, and a fan's constants are bounded by the masks that
differ."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from code_mojo_gb300 import butterfly as bfy
from code_mojo_gb300 import workloads as W
from oracle import pyoracle as O
from tests.test_phase_fans import model, phase_mix, run_model  # noqa: F401 (model: a fixture)

ROOT = Path(__file__).resolve().parent.parent
CUDA_INC = Path("/usr/local/cuda/include")


@pytest.fixture(scope="module")
def depth(tmp_path_factory):
    if shutil.which("g++") is None or not CUDA_INC.exists():
        pytest.skip("needs g++ and the CUDA headers")
    from code_mojo_gb300 import build
    lib = build.build_engine()
    exe = tmp_path_factory.mktemp("fan_depth") / "fan_depth"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(CUDA_INC), "-I", str(ROOT / "include"),
                    str(ROOT / "tests" / "fan_depth.cpp"), "-o", str(exe), "-L", str(lib.parent), "-lbfgpu",
                    f"-Wl,-rpath,{lib.parent}"], check=True, capture_output=True)
    return exe


def alternating(n, count, qubits):
    """Phases on the given qubits in turn, each after a dense gate on qubit 0."""
    qc = bfy.QuantumCircuit(n)
    for k in range(count // 2):
        qc.u3(0, 0.1 * k, 0.3, 0.2)
        q = qubits[k % len(qubits)]
        if isinstance(q, tuple):
            qc.cp(q[0], q[1], 0.01 * (k + 1))
        else:
            qc.p(q, 0.01 * (k + 1))
    return qc


def plan(depth, qc, K, units, tmp_path):
    ops = tmp_path / "ops.bin"
    ops.write_bytes(bfy.serialize(qc))
    best = None
    for _ in range(3):
        r = subprocess.run([str(depth), str(ops), str(K), str(units)], check=True, capture_output=True, text=True)
        f = r.stdout.split()
        best = [int(x) for x in f[:3]] + [min(float(f[3]), best[3] if best else 1e9)]
    return best  # ops, fans, most constants, ms


# phases outside the tile, inside it, and with a control outside; with tensor
# blocks in view the cost estimate scans the phases as well
@pytest.mark.parametrize("qubits", [[12, 13], [5, 6, 11], [(3, 12), (4, 13), (13, 2)]])
@pytest.mark.parametrize("units", [0, 2.5])
def test_planning_time_grows_with_the_gate_count(depth, qubits, units, tmp_path):
    few = plan(depth, alternating(14, 5000, qubits), 12, units, tmp_path)
    many = plan(depth, alternating(14, 40000, qubits), 12, units, tmp_path)
    # eight times the gates; a rescan of every waiting phase takes 64 times as long
    assert many[3] <= 20 * few[3] + 20
    for ops, fans, most, _ in (few, many):
        assert most <= len(qubits)
    assert many[0] <= 20000 + 64  # the dense gates, and what the merged phases leave


def test_repeated_masks_match_the_oracle(model, tmp_path):  # noqa: F811
    for qubits in ([6, 1], [2, (3, 6), (6, 3), 2, 2], [(1, 2), (2, 1), 5]):
        qc = alternating(7, 400, qubits)
        re, im = W.random_normal_state(7, 3)
        for K in (6, 7):
            got, _ = run_model(model, qc, re, im, K, 0, tmp_path)
            r, i = O.run(qc, re, im)
            assert np.max(np.abs(got - (r + 1j * i))) <= 4 * 400 * 2.0 ** -53  # a few roundings of 2^-53 per op


def many_constant_fans(n, gates):
    """A fan with a constant from outside the tile before each dense gate on
    qubit 0 (the gates keep qubits 0 to 5 in a 6-qubit tile, and n-1 out of it)."""
    qc = bfy.QuantumCircuit(n)
    for k in range(gates):
        qc.cp(n - 1, 0, 0.01 * (k + 1))
        qc.cp(1 + k % 5, 0, 0.02 * (k + 1))
        qc.u3(0, 0.1 * k, 0.3, 0.2)
        qc.ry(1 + k % 5, 0.3)
    return qc


DEEP = {"mix": (9, 11, lambda: phase_mix(9, 2500, 5)), "mix_tiles": (12, 7, lambda: phase_mix(12, 1500, 6)),
        "constants": (8, 6, lambda: many_constant_fans(8, 150))}


# more fans than a pass has slots for constants: those without constants need
# none, and phases from outside the tile stay ops once the slots are taken
@pytest.mark.parametrize("name", list(DEEP))
def test_more_fans_than_constants(model, name, tmp_path):  # noqa: F811
    n, K, make = DEEP[name]
    qc = make()
    re, im = W.random_normal_state(n, 4)
    got, (tiles, _, fans, phases) = run_model(model, qc, re, im, K, 0, tmp_path)
    r, i = O.run(qc, re, im)
    assert np.max(np.abs(got - (r + 1j * i))) <= 4 * len(qc.transformations) * 2.0 ** -53
    if name == "constants":
        assert fans == 64 and phases >= 150 - 64
    else:
        assert fans > 64 and (name != "mix" or tiles == 1)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("name", list(DEEP))
def test_more_fans_than_constants_on_the_gpu(name, dtype):
    n, K, make = DEEP[name]
    qc = make()
    re, im = W.random_normal_state(n, 4)
    ctx = bfy.ExecContext()
    ctx.gpu_tile_qubits = K
    st = bfy.QuantumState.from_soa(re, im, dtype)
    bfy.execute(st, qc, ctx)
    got = st.to_complex()
    st.close()
    r, i = O.run(qc, re, im)
    exp = r + 1j * i
    # a few roundings per op: 2^-46 in a double-float pair, 2^-24 in FP32
    unit = 2.0 ** -46 if dtype == "c128" else 2.0 ** -24
    assert np.linalg.norm(got - exp) <= 4 * len(qc.transformations) * unit
