"""The work a user of this engine has it do, as timed cases.

Each case is one call sequence through the package's public entry points
(QuantumState, execute, Batch, Server): a circuit run on a state that stays on
the GPU, and the readout a program of that kind does with the result.  The
circuits are described here as plain tuples, from which both the package's
circuit objects and the 64-bit evaluation of `exact` are made.
"""
import ctypes
import math

import numpy as np
import torch

from code_mojo_gb300 import butterfly as bfy
from code_mojo_gb300 import opsarray
from code_mojo_gb300.batch import Batch
from code_mojo_gb300.serving import Server


def listed():
    return [
        # A small circuit submitted as Python objects, state in and state out:
        # what an interactive session or a unit test does (launch latency).
        {"name": "encode_9q_c128_object", "kind": "encode", "n": 9, "dtype": "c128", "strategy": "fused",
         "source": "object", "start": "upload", "read": "state"},
        # The 20-qubit QFT of a dense random state, kept on the device, the
        # spectrum read back.
        {"name": "qft_20q_c128", "kind": "qft", "n": 20, "dtype": "c128", "strategy": "fused",
         "source": "list", "start": "resident", "read": "state"},
        # The reference's published benchmark circuit (value encoding) at its
        # largest published size, from |0>, read out as a register distribution.
        {"name": "encode_24q_c128", "kind": "encode", "n": 24, "dtype": "c128", "strategy": "fused",
         "source": "list", "start": "zero", "read": "probs", "reg": 20},
        # The same family in single precision, large state.
        {"name": "encode_27q_c64", "kind": "encode", "n": 27, "dtype": "c64", "strategy": "fused",
         "source": "list", "start": "zero", "read": "probs", "reg": 12},
        # Random layered circuits (U3 on every qubit, CX matching per layer):
        # the headline workload family, dense gates, complex128.
        {"name": "layered_28q_c128", "kind": "layered", "n": 28, "layers": 20, "dtype": "c128", "strategy": "fused",
         "source": "list", "start": "zero", "read": "probs", "reg": 16},
        # ... in single precision.
        {"name": "layered_29q_c64", "kind": "layered", "n": 29, "layers": 16, "dtype": "c64", "strategy": "fused",
         "source": "list", "start": "zero", "read": "probs", "reg": 16},
        # Gate-by-gate execution (no fusion), the whole state read back: the
        # per-gate strategy that a program checking each step or porting from
        # the reference's scalar strategies uses.
        {"name": "gates_24q_c128", "kind": "layered", "n": 24, "layers": 3, "dtype": "c128", "strategy": "gate",
         "source": "list", "start": "zero", "read": "state"},
        # Grover search with the classical oracle and diffuser, full iteration
        # count, outcome distribution over every qubit.
        {"name": "grover_20q_c128", "kind": "grover", "n": 20, "dtype": "c128", "strategy": "fused",
         "source": "list", "start": "zero", "read": "probs", "reg": 20},
        # Shor order finding: modular exponentiation, then the inverse QFT on
        # the exponent register, whose distribution is what the caller needs.
        {"name": "order_24q_c128", "kind": "order", "n": 24, "n_value": 8, "dtype": "c128", "strategy": "fused",
         "source": "list", "start": "zero", "read": "probs", "reg": 16},
        # Many independent small circuits in one launch, every state read back:
        # half random layered circuits of depth 20, half value encodings.
        {"name": "batch_128x8-16q_c64", "kind": "batch", "count": 128, "nmin": 8, "nmax": 16, "depth": 20,
         "dtype": "c64"},
        {"name": "batch_48x10-17q_c128", "kind": "batch", "count": 48, "nmin": 10, "nmax": 17, "depth": 20,
         "dtype": "c128"},
        # Serving: a burst of requests (Grover, value encoding, layered) from
        # submission to the last result.
        {"name": "serve_36x10-20q_c128", "kind": "serve", "count": 36, "nmin": 10, "nmax": 20, "dtype": "c128"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["encode", "encode", "qft", "layered", "layered", "gates", "grover", "order", "batch", "serve"])
    dtype = rng.choice(["c128", "c64"])
    if kind == "batch":
        top = rng.randint(10, 16 if dtype == "c64" else 15)
        return {"kind": "batch", "count": _log_int(rng, 8, 96), "nmin": rng.randint(5, 9), "nmax": top,
                "depth": rng.randint(3, 24), "dtype": dtype}
    if kind == "serve":
        return {"kind": "serve", "count": _log_int(rng, 4, 32), "nmin": rng.randint(8, 12), "nmax": rng.randint(14, 20),
                "dtype": "c128"}
    case = {"kind": "layered" if kind == "gates" else kind, "dtype": dtype,
            "strategy": "gate" if kind == "gates" else "fused", "source": "list", "start": "zero", "read": "probs"}
    if kind == "encode":
        case["n"] = rng.randint(7, 24 if dtype == "c128" else 27)
    elif kind == "qft":
        case["n"] = rng.randint(7, 22)
        case["start"] = "resident"
    elif kind == "layered":
        case["n"] = rng.randint(8, 27 if dtype == "c128" else 28)
        case["layers"] = rng.randint(2, 16)
    elif kind == "gates":
        case["n"] = rng.randint(8, 25)
        case["layers"] = rng.randint(1, 2)
    elif kind == "grover":
        case["n"] = rng.randint(8, 20)
    else:
        case["n_value"] = rng.randint(4, 9)
        case["n"] = case["n_value"] + rng.randint(6, 16)
    if case["n"] <= 21 and case["kind"] != "grover" and rng.random() < 0.5:
        case["read"] = "state"
        if case["n"] <= 14 and rng.random() < 0.5:
            case["source"], case["start"] = "object", "upload"
    else:
        case["reg"] = case["n"] - case["n_value"] if kind == "order" else rng.randint(3, min(20, case["n"]))
    return case


# ---- circuits as plain tuples ------------------------------------------------


def _rng(*key):
    return np.random.Generator(np.random.PCG64([int(k) for k in key]))


def _iqft(qubits):
    """Inverse QFT, first listed qubit last: H, then the controlled phases."""
    ops = []
    for j in reversed(range(len(qubits))):
        ops.append(("h", qubits[j]))
        for k in reversed(range(j)):
            ops.append(("cp", qubits[j], qubits[k], -math.pi / 2 ** (j - k)))
    return ops


def _encode(n, v):
    """H on all qubits, the phases of the value v, the inverse QFT."""
    ops = [("h", j) for j in range(n)]
    ops += [("p", j, 2 * math.pi / 2 ** (j + 1) * v) for j in range(n)]
    return ops + _iqft([n - 1 - j for j in range(n)])


def _layered(n, layers, rng):
    ops = []
    for _ in range(layers):
        a = rng.uniform(0.0, 2 * math.pi, size=(n, 3))
        ops += [("u3", q, float(a[q, 0]), float(a[q, 1]), float(a[q, 2])) for q in range(n)]
        perm = rng.permutation(n)
        ops += [("cx", int(perm[k]), int(perm[k + 1])) for k in range(0, n - 1, 2)]
    return ops


def _iterations(n):
    return int(math.floor(math.pi / 4 * math.sqrt(2 ** n)))


def _modulus(case, rng):
    """A modulus that fills the value register and a base coprime to it."""
    top = 1 << case["n_value"]
    mod = int(rng.integers(top // 2 + 1, top))
    while True:
        a = int(rng.integers(2, mod))
        if math.gcd(a, mod) == 1:
            return a, mod


def _circuit(case, seed):
    rng = _rng(seed, 1)
    n, kind = case["n"], case["kind"]
    if kind == "encode":
        return _encode(n, float(rng.uniform(0, 2 ** min(n, 20))))
    if kind == "qft":
        fwd = []
        for op in reversed(_iqft([n - 1 - j for j in range(n)])):
            fwd.append(op if op[0] == "h" else ("cp", op[1], op[2], -op[3]))
        return fwd + [("bitrev",)]
    if kind == "layered":
        return _layered(n, case["layers"], rng)
    if kind == "grover":
        return [("h", q) for q in range(n)] + [("search", int(rng.integers(0, 2 ** n)), _iterations(n))]
    n_exp = n - case["n_value"]
    a, mod = _modulus(case, rng)
    ops = [("h", q) for q in range(n_exp)] + [("x", n_exp), ("modexp", n_exp, case["n_value"], a, mod)]
    return ops + _iqft([n_exp - 1 - j for j in range(n_exp)])


def _package_circuit(n, ops):
    """The tuples as the package's circuit object (an op array for a search)."""
    if ops[-1][0] == "search":
        return opsarray.grover(n, ops[-1][1], ops[-1][2])
    qc = bfy.QuantumCircuit(n)
    for op in ops:
        name = op[0]
        if name == "h":
            qc.h(op[1])
        elif name == "x":
            qc.x(op[1])
        elif name == "p":
            qc.p(op[1], op[2])
        elif name == "cp":
            qc.cp(op[1], op[2], op[3])
        elif name == "cx":
            qc.cx(op[1], op[2])
        elif name == "u3":
            qc.u3(op[1], op[2], op[3], op[4])
        elif name == "bitrev":
            bfy.bit_reverse(qc)
        else:
            bfy.mod_exp(qc, op[1], op[2], op[3], op[4])
    return qc


def _spread(i):
    """Positions 0, 1, ... spread evenly over [0, 1): the sizes of a mix."""
    return (i + 1) * 0.6180339887498949 % 1.0


def _requests(case, seed):
    """The served mix: (kind, n, ops) in turn Grover, value encoding, layered."""
    rng = _rng(seed, 2)
    out = []
    for i in range(case["count"]):
        n = round(case["nmin"] * (case["nmax"] / case["nmin"]) ** _spread(i))
        if i % 3 == 0:
            out.append((n, [("h", q) for q in range(n)] + [("search", int(rng.integers(0, 2 ** n)), _iterations(n))]))
        elif i % 3 == 1:
            out.append((n, _encode(n, float(rng.uniform(0, 2 ** n)))))
        else:
            out.append((n, _layered(n, int(rng.integers(10, 41)), rng)))
    return out


def _members(case, seed):
    """The batch: even positions layered, odd ones value encodings."""
    rng = _rng(seed, 3)
    out = []
    for i in range(case["count"]):
        n = case["nmin"] + int(_spread(i) * (case["nmax"] + 1 - case["nmin"]))
        out.append((n, _layered(n, case["depth"], rng) if i % 2 == 0 else _encode(n, float(rng.uniform(0, 2 ** n)))))
    return out


def _dense_state(n, seed):
    rng = _rng(seed, 4)
    re, im = rng.standard_normal(1 << n), rng.standard_normal(1 << n)
    s = math.sqrt(float(re @ re + im @ im))
    return re / s, im / s


def _register(case, seed):
    """The qubits read out: the exponent register, or a seeded choice."""
    if case["kind"] == "order":
        return list(range(case["reg"]))
    return sorted(int(q) for q in _rng(seed, 5).permutation(case["n"])[:case["reg"]])


# ---- the framework's side -----------------------------------------------------


def _op_array(circuit):
    """A circuit flattened once, as a program that submits it often keeps it."""
    arr, count, keep = circuit.to_ops()
    raw = np.frombuffer(ctypes.string_at(ctypes.addressof(arr), count * 128), dtype=opsarray.BF_OP).copy()
    return opsarray.OpArray(circuit.num_qubits, raw, [arr, keep])


def prepare(case, seed):
    if case["kind"] == "batch":
        return {"case": case, "batch": Batch([_package_circuit(n, ops) for n, ops in _members(case, seed)], case["dtype"])}
    if case["kind"] == "serve":
        reqs = []
        for n, ops in _requests(case, seed):
            c = _package_circuit(n, ops)
            reqs.append(c if isinstance(c, opsarray.OpArray) else _op_array(c))
        return {"case": case, "server": Server(), "requests": reqs}
    n = case["n"]
    circuit = _package_circuit(n, _circuit(case, seed))
    if case["source"] == "list" and not isinstance(circuit, opsarray.OpArray):
        circuit = bfy.deserialize(bfy.serialize(circuit))
    ctx = bfy.ExecContext()
    ctx.execution_strategy = bfy.ExecutionStrategy.GPU if case["strategy"] == "gate" else bfy.ExecutionStrategy.GPU_FUSED
    ctx.gpu_sync = False
    st = {"case": case, "circuit": circuit, "ctx": ctx}
    if case["start"] == "upload":
        st["host"] = _dense_state(n, seed)
        st["state"] = bfy.QuantumState(n, case["dtype"])
    elif case["start"] == "resident":
        st["state"] = bfy.QuantumState.from_soa(*_dense_state(n, seed), case["dtype"])
    else:
        st["state"] = bfy.QuantumState(n, case["dtype"])
    if case["read"] == "probs":
        st["register"] = _register(case, seed)
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "batch":
        b = st["batch"]
        b.run(sync=False)
        z = np.concatenate([b.download(c) for c in range(case["count"])])
        return z.astype(np.complex64) if case["dtype"] == "c64" else z
    if case["kind"] == "serve":
        srv = st["server"]
        ids = [srv.submit(r, case["dtype"]) for r in st["requests"]]
        srv.wait_idle(60.0)
        by = {r.id: r for r in srv.poll()}
        return {"index": np.concatenate([by[i].top_index for i in ids]).astype(np.int64),
                "prob": np.concatenate([by[i].top_prob for i in ids])}
    state = st["state"]
    if case["start"] == "upload":
        state.upload(*st["host"])
    elif case["start"] == "zero":
        state.set_basis(0)
    bfy.execute(state, st["circuit"], st["ctx"])
    kind = np.float64 if case["dtype"] == "c128" else np.float32
    if case["read"] == "state":
        return [x.astype(kind, copy=False) for x in state.download()]
    return state.probabilities(st["register"]).astype(kind, copy=False)


# ---- what a pass cannot do without --------------------------------------------


def _flops(n, ops):
    """Floating-point operations of the gates applied one by one."""
    amps, f = 2.0 ** n, 0.0
    for op in ops:
        if op[0] == "u3":
            f += 14 * amps
        elif op[0] == "h":
            f += 4 * amps
        elif op[0] == "p":
            f += 3 * amps
        elif op[0] == "cp":
            f += 1.5 * amps
        elif op[0] == "search":
            f += 4 * amps  # the iterations compose to one affine map
    return f


def work(case):
    size = 16 if case["dtype"] == "c128" else 8
    if case["kind"] == "batch":
        members = _members(case, 0)
        return {"bytes": sum(size * 2.0 ** n + 16 * 2.0 ** n for n, _ in members),
                "flops": sum(_flops(n, ops) for n, ops in members)}
    if case["kind"] == "serve":
        members = _requests(case, 0)
        return {"bytes": sum(2.0 * size * 2.0 ** n for n, _ in members), "flops": sum(_flops(n, ops) for n, ops in members)}
    amps = 2.0 ** case["n"]
    read = 16 * amps if case["read"] == "state" else 8 * 2.0 ** case["reg"]
    return {"bytes": 2.0 * size * amps + read, "flops": _flops(case["n"], _circuit(case, 0))}


# ---- the same in plain torch, 64 bits ------------------------------------------


def _apply(psi, n, op):
    """One op on a complex128 vector, in place where it can be."""
    name = op[0]
    if name == "bitrev":
        return psi.view([2] * n).permute(list(reversed(range(n)))).reshape(-1)
    if name == "modexp":
        _, n_exp, n_value, a, mod = op
        v = psi.view(1 << n_value, 1 << n_exp)
        x = [pow(a, e, mod) for e in range(1 << n_exp)]
        mult = torch.tensor(x, device=psi.device)
        y = torch.arange(1 << n_value, device=psi.device)[:, None]
        dst = torch.where(y < mod, y * mult[None, :] % mod, y.expand(-1, 1 << n_exp))
        return torch.zeros_like(v).scatter_(0, dst, v).reshape(-1)
    if name == "search":
        _, marked, count = op
        for _ in range(count):
            psi[marked] = -psi[marked]
            psi = 2 * psi.mean() - psi
        return psi
    if name in ("cp", "cx"):
        hi, lo = max(op[1], op[2]), min(op[1], op[2])
        v = psi.view(1 << (n - 1 - hi), 2, 1 << (hi - lo - 1), 2, 1 << lo)
        if name == "cp":
            v[:, 1, :, 1, :] *= complex(math.cos(op[3]), math.sin(op[3]))
        else:
            one = v[:, 1] if op[1] == hi else v[:, :, :, 1]
            pair = (one[:, :, 0], one[:, :, 1]) if op[1] == hi else (one[:, 0], one[:, 1])
            keep = pair[0].clone()
            pair[0].copy_(pair[1])
            pair[1].copy_(keep)
        return psi
    v = psi.view(1 << (n - 1 - op[1]), 2, 1 << op[1])
    if name == "p":
        v[:, 1, :] *= complex(math.cos(op[2]), math.sin(op[2]))
        return psi
    if name == "x":
        return v.flip(1).reshape(-1)
    a, b = v[:, 0, :].clone(), v[:, 1, :]
    if name == "h":
        s = math.sqrt(0.5)
        v[:, 0, :] = (a + b) * s
        v[:, 1, :] = a * s - (v[:, 0, :] - a * s)
        return psi
    _, _, theta, phi, lam = op
    c, s = math.cos(theta / 2), math.sin(theta / 2)
    el, ep = complex(math.cos(lam), math.sin(lam)), complex(math.cos(phi), math.sin(phi))
    m11 = complex(math.cos(phi + lam), math.sin(phi + lam)) * c
    new = a * c - b * (el * s)
    b.mul_(m11).add_(a * (ep * s))
    v[:, 0, :] = new
    return psi


def _evolve(n, ops, start=None):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if start is None:
        psi = torch.zeros(1 << n, dtype=torch.complex128, device=dev)
        psi[0] = 1
    else:
        psi = torch.complex(torch.from_numpy(start[0]), torch.from_numpy(start[1])).to(dev)
    for op in ops:
        psi = _apply(psi, n, op)
    return psi


def exact(case, seed):
    if case["kind"] == "batch":
        return torch.cat([_evolve(n, ops) for n, ops in _members(case, seed)]).cpu().numpy()
    if case["kind"] == "serve":
        probs = []
        for n, ops in _requests(case, seed):
            p = _evolve(n, ops).abs().square()
            probs.append(torch.topk(p, 16).values)
        return {"index": None, "prob": torch.cat(probs).cpu().numpy()}
    n = case["n"]
    psi = _evolve(n, _circuit(case, seed), None if case["start"] == "zero" else _dense_state(n, seed))
    if case["read"] == "state":
        return [psi.real.cpu().numpy(), psi.imag.cpu().numpy()]
    keep = _register(case, seed)
    p = psi.abs().square()
    # sum the other qubits out, from the highest down
    for q in reversed(range(n)):
        if q not in keep:
            p = p.view(-1, 2, 1 << q).sum(1).reshape(-1)
    return p.cpu().numpy()
