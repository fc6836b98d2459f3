"""The dense statevector engine's measured workloads.

Each case is one call sequence a program makes through the package's public
entry points: whole jobs through ``B200DenseEngine.execute``, program sweeps
on a device state in both precisions, Pauli expectations and sampling of a
state the program holds, batched parameter sweeps, a burst through the
serving loop, and the two noisy engines.  Circuits are the families of
``menos_b200.workloads`` with angles drawn from the seed.

``exact`` evolves the same circuits gate by gate in plain complex128 torch.
"""
import math

import numpy as np
import torch

from menos_b200 import Context, DeviceState, workloads
from menos_b200._lib import C64, C128
from menos_b200.circuit import OP, Circuit, PackedCircuit
from menos_b200.engine import (B200DenseEngine, DensityMatrix, EngineExecutionRequest, PauliTerm, sweep_batch,
                               trajectories)
from menos_b200.serve import Server

_CONTEXT = None


def _context():
    """One context per process, as a program holds it."""
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = Context(0)
    return _CONTEXT


def listed():
    return [
        # A small job: latency, launches and host work count.
        {"name": "job_12q", "kind": "job", "qubits": 12, "depth": 8, "qft": False, "paulis": 16, "shots": 1024,
         "statevector": True},
        # 20 qubits, 20 layers, statevector and 4096 shots: workloads.config_c1.
        {"name": "job_20q", "kind": "job", "qubits": 20, "depth": 20, "qft": False, "paulis": 0, "shots": 4096,
         "statevector": True},
        # The headline job (brick depth 40, QFT, 64 Pauli strings, 1e6 shots) four qubits below its 30.
        {"name": "job_26q", "kind": "job", "qubits": 26, "depth": 40, "qft": True, "paulis": 64, "shots": 1000000,
         "statevector": False},
        # The headline's state size: 16 GiB of complex128, fewer layers.
        {"name": "sweep_30q", "kind": "sweep", "qubits": 30, "depth": 12, "family": "brick", "precision": "c128"},
        # The precision path below and above the size where it turns to the tensor cores.
        {"name": "sweep_c64_23q", "kind": "sweep", "qubits": 23, "depth": 20, "family": "hea", "precision": "c64"},
        {"name": "sweep_c64_28q", "kind": "sweep", "qubits": 28, "depth": 20, "family": "brick", "precision": "c64"},
        # An observable of 64 Pauli strings, and 1e6 shots, of a state the program holds.
        {"name": "paulis_27q", "kind": "paulis", "qubits": 27, "terms": 64, "precision": "c128"},
        {"name": "sample_27q", "kind": "sample", "qubits": 27, "shots": 1000000, "precision": "c128"},
        # A variational step: <H> for many bindings of one ansatz (bench.py --mode batch, an eighth of its rows).
        {"name": "bindings_16q", "kind": "bindings", "qubits": 16, "layers": 8, "bindings": 512, "terms": 32,
         "precision": "c128"},
        # A burst of small requests into the serving loop.
        {"name": "serve_12_16q", "kind": "serve", "requests": 128, "lowest": 12, "highest": 16},
        # Noisy circuits: the density matrix (a 22-qubit state) and trajectories.
        {"name": "density_11q", "kind": "density", "qubits": 11, "depth": 4, "terms": 16, "shots": 4096},
        {"name": "trajectories_14q", "kind": "trajectories", "qubits": 14, "depth": 3, "count": 8, "terms": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["job", "sweep", "sweep", "paulis", "sample", "bindings", "serve", "density", "trajectories"])
    if kind == "job":
        n = rng.randint(9, 26)
        qft = rng.random() < 0.5
        return {"kind": kind, "qubits": n, "depth": _log_int(rng, 4, 40), "qft": qft, "paulis": rng.randint(1, 64),
                "shots": _log_int(rng, 100, 1000000), "statevector": n <= 20}
    if kind == "sweep":
        n = rng.randint(13, 30)
        return {"kind": kind, "qubits": n, "depth": _log_int(rng, 4, 40 if n < 27 else 20 if n < 29 else 10),
                "family": rng.choice(["brick", "hea"] if n < 29 else ["brick"]),
                "precision": rng.choice(["c128", "c64"])}
    if kind == "paulis":
        return {"kind": kind, "qubits": rng.randint(10, 28), "terms": _log_int(rng, 1, 64),
                "precision": rng.choice(["c128", "c128", "c64"])}
    if kind == "sample":
        return {"kind": kind, "qubits": rng.randint(10, 28), "shots": _log_int(rng, 100, 1000000),
                "precision": rng.choice(["c128", "c128", "c64"])}
    if kind == "bindings":
        n = rng.randint(8, 16)
        most = min(2048, 512 << (16 - n))
        return {"kind": kind, "qubits": n, "layers": rng.randint(2, 8), "bindings": _log_int(rng, 16, most),
                "terms": rng.randint(4, 48), "precision": rng.choice(["c128", "c64"])}
    if kind == "serve":
        low = rng.randint(10, 14)
        return {"kind": kind, "requests": _log_int(rng, 8, 160), "lowest": low, "highest": low + rng.randint(0, 4)}
    if kind == "density":
        return {"kind": kind, "qubits": rng.randint(5, 11), "depth": rng.randint(2, 5), "terms": rng.randint(1, 16),
                "shots": _log_int(rng, 100, 10000)}
    return {"kind": kind, "qubits": rng.randint(6, 16), "depth": rng.randint(1, 4), "count": rng.randint(2, 12),
            "terms": rng.randint(1, 12)}


# ---------------------------------------------------------------- inputs
def _depolarizing(p):
    x, y, z = np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]), np.diag([1, -1])
    return np.array([math.sqrt(1 - p) * np.eye(2)] + [math.sqrt(p / 3) * m for m in (x, y, z)], np.complex128)


def _damping(g):
    return np.array([[[1, 0], [0, math.sqrt(1 - g)]], [[0, math.sqrt(g)], [0, 0]]], np.complex128)


def _noisy(n, depth, seed):
    """Brick layers, each followed by depolarizing noise on every qubit and amplitude damping on every third."""
    layers = workloads.brick(n, depth, seed).ops
    c = Circuit(n)
    cz = OP["cz"]
    for i, op in enumerate(layers):
        c.ops.append(op)
        if op[0] == cz and (i + 1 == len(layers) or layers[i + 1][0] != cz):
            for q in range(n):
                c.channel([q], _depolarizing(0.01) if q % 3 else _damping(0.02))
    return c


def _circuit(case, seed):
    kind = case["kind"]
    if kind == "job":
        c = workloads.brick(case["qubits"], case["depth"], seed)
        return workloads.qft(case["qubits"], c) if case["qft"] else c
    if kind == "sweep":
        return getattr(workloads, case["family"])(case["qubits"], case["depth"], seed)
    if kind in ("paulis", "sample"):
        return workloads.brick(case["qubits"], 5, seed)
    if kind == "bindings":
        return workloads.hea(case["qubits"], case["layers"], seed)
    return _noisy(case["qubits"], case["depth"], seed)


def _stream(case, seed):
    return workloads.serving_stream(case["requests"], 1.0, seed, nmin=case["lowest"], nmax=case["highest"])


def _precision(case):
    return C64 if case["precision"] == "c64" else C128


class _Amplitudes:
    """A device state's memory for torch (it keeps the state alive)."""

    def __init__(self, state):
        import ctypes
        from menos_b200._lib import lib
        p = ctypes.c_void_p()
        assert lib().mb2_state_device_ptr(state.h, ctypes.byref(p)) == 0
        self.state = state
        self.__cuda_array_interface__ = {"shape": (1 << state.n, 2), "data": (p.value, False), "version": 3,
                                         "typestr": "<f8" if state.precision == C128 else "<f4"}


def _amplitudes(state):
    return torch.as_tensor(_Amplitudes(state), device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    ctx = _context()
    if kind == "serve":
        s["requests"] = _stream(case, seed)
        for r in s["requests"]:
            r["circuit"] = PackedCircuit(r["circuit"])
        s["server"] = Server(ctx, budget_bytes=20 * 10 ** 9)
        s["shots"] = 4096 * len(s["requests"])
        return s
    n = case["qubits"]
    circ = _circuit(case, seed)
    s["circuit"] = circ
    s["shots"] = case.get("shots", 0)
    if kind == "job":
        s["engine"] = B200DenseEngine(0)
        s["request"] = EngineExecutionRequest(
            n, circ, want_statevector=case["statevector"], want_counts=True, want_expectation=case["paulis"] > 0,
            shots=case["shots"], measure_targets=[(q, q) for q in range(n)], bitstring_width=n, seed=seed,
            observable=[PauliTerm(x, z) for x, z in workloads.pauli_strings(n, case["paulis"], seed + 1)])
    elif kind == "sweep":
        s["state"] = DeviceState(ctx, n, _precision(case))
        s["amplitudes"] = _amplitudes(s["state"])
    elif kind in ("paulis", "sample"):
        s["state"] = DeviceState(ctx, n, _precision(case))
        s["state"].init()
        s["state"].apply_program(circ)
        s["seed"] = seed + 2
        s["targets"] = [(q, q) for q in range(n)]
        if kind == "paulis":
            s["paulis"] = workloads.pauli_strings(n, case["terms"], seed + 1)
    elif kind == "bindings":
        s["params"] = np.random.default_rng(seed).uniform(-math.pi, math.pi, (case["bindings"], 2 * n * case["layers"]))
        s["paulis"] = workloads.pauli_strings(n, case["terms"], seed + 1)
        s["coefs"] = workloads.weights(case["terms"], seed + 2)
    else:
        s["paulis"] = workloads.pauli_strings(n, case["terms"], seed + 1)
        s["seed"] = seed + 2
        if kind == "density":
            s["rho"] = DensityMatrix(ctx, n)
            s["amplitudes"] = _amplitudes(s["rho"].state)
            s["targets"] = [(q, q) for q in range(n)]
    return s


# ---------------------------------------------------------------- the call
def _keep(s, name, arrays, size):
    """The arrays one after another at the head of a buffer of the state's that holds one value per shot."""
    buf = s.setdefault(name, np.zeros(size, np.uint64))
    at = 0
    for a in arrays:
        buf[at:at + len(a)] = a
        at += len(a)
    buf[at:] = 0
    return buf.view(np.int64)


def _counts(s, counts):
    """Outcomes and counts of one sampling call (or of several), as arrays whose size does not depend on the
    draw."""
    counts = counts if isinstance(counts, list) else [counts]
    return {"outcomes": _keep(s, "outcomes", [c.outcomes for c in counts], s["shots"]),
            "counts": _keep(s, "counts", [c.counts for c in counts], s["shots"])}


def _serve(s):
    server, at, values, counts = s["server"], {}, {}, {}
    for i, r in enumerate(s["requests"]):
        if r["output"] == "counts":
            n = r["circuit"].num_qubits
            t = server.submit(r["circuit"], "counts", shots=r["shots"], seed=r["seed"],
                              targets=[(q, q) for q in range(n)])
        else:
            t = server.submit(r["circuit"], "expectation", paulis=r["paulis"], coefs=r["coefs"])
        at[t] = i
    left = len(at)
    while left:
        for c in server.poll(timeout_ms=100):
            if c["status"] != 0:
                raise RuntimeError("request %d: status %d" % (at[c["ticket"]], c["status"]))
            if s["requests"][at[c["ticket"]]]["output"] == "counts":
                counts[at[c["ticket"]]] = c["counts"]
            else:
                values[at[c["ticket"]]] = c["value"]
            left -= 1
    return {"values": np.array([values.get(i, 0.0) for i in range(len(at))]),
            "sample": _counts(s, [counts[i] for i in sorted(counts)])}


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "job":
        r = s["engine"].execute(s["request"])
        return {"state": r.statevector, "terms": r.expectation_terms, "sample": _counts(s, r.counts)}
    if kind == "sweep":
        s["state"].init()
        s["state"].apply_program(s["circuit"])
        if case["precision"] == "c64":
            s["state"].normalize()
        return s["amplitudes"]
    if kind == "paulis":
        return s["state"].expectation(s["paulis"])
    if kind == "sample":
        return _counts(s, s["state"].sample(case["shots"], s["seed"], s["targets"]))
    if kind == "bindings":
        return sweep_batch(_context(), s["circuit"], s["params"], s["paulis"], s["coefs"],
                           precision=_precision(case))[0]
    if kind == "serve":
        return _serve(s)
    if kind == "density":
        s["rho"].init()
        s["rho"].apply(s["circuit"])
        return {"rho": s["amplitudes"], "terms": s["rho"].expectation(s["paulis"]),
                "sample": _counts(s, s["rho"].sample(case["shots"], s["seed"], s["targets"]))}
    r = trajectories(_context(), s["circuit"], case["count"], s["seed"], s["paulis"])
    return {"terms": r["terms"], "standard_error": r["standard_error"]}


# ---------------------------------------------------------------- what it cannot do without
def _gate_flops(ops):
    """Real operations per amplitude: a dense complex 2x2 is two products and a sum, a real one on complex
    amplitudes half of that; diagonals multiply the amplitudes whose entry is not one; signs and
    permutations are free."""
    per = {OP["u"]: 14.0, OP["h"]: 6.0, OP["ry"]: 6.0, OP["rz"]: 6.0, OP["cp"]: 1.5}
    return sum(per.get(op[0], 0.0) for op in ops)


def work(case):
    kind = case["kind"]
    if kind == "serve":
        bytes_, flops = 0.0, 0.0
        for r in _stream(case, 1):
            n = r["circuit"].num_qubits
            flops += 2.0 ** n * (_gate_flops(r["circuit"].ops) + (4 if r["output"] == "counts" else 6 * 32))
            bytes_ += 48.0 * len(r["circuit"].ops) + (16 * 4096 if r["output"] == "counts" else 8)
        return {"bytes": bytes_, "flops": flops}
    n = case["qubits"]
    amp = 8 if case.get("precision") == "c64" else 16
    ops = _circuit(case, 1).ops
    if kind == "job":
        return {"bytes": amp * 2.0 ** n + 16.0 * case["shots"],
                "flops": 2.0 ** n * (_gate_flops(ops) + 6 * case["paulis"] + 4)}
    if kind == "sweep":
        return {"bytes": amp * 2.0 ** n, "flops": 2.0 ** n * _gate_flops(ops)}
    if kind == "paulis":
        return {"bytes": amp * 2.0 ** n, "flops": 2.0 ** n * 6 * case["terms"]}
    if kind == "sample":
        return {"bytes": amp * 2.0 ** n + 16.0 * case["shots"], "flops": 2.0 ** n * 4}
    if kind == "bindings":
        b = case["bindings"]
        return {"bytes": 8.0 * b * (2 * n * case["layers"] + 1),
                "flops": b * 2.0 ** n * (_gate_flops(ops) + 6 * case["terms"])}
    channels = sum(op[0] == OP["channel"] for op in ops)
    if kind == "density":  # U on the rows and on the columns; a channel's 4x4 superoperator on (row, column)
        return {"bytes": 16.0 * 4.0 ** n, "flops": 4.0 ** n * (2 * _gate_flops(ops) + 30 * channels)}
    return {"bytes": 48.0 * len(ops) + 16.0 * case["terms"],
            "flops": case["count"] * 2.0 ** n * (_gate_flops(ops) + 30 * channels + 6 * case["terms"])}


def tolerance(case):
    kind = case["kind"]
    # A complex128 state is defined to the bit (each amplitude sees its gates in plan order, every product
    # and sum rounded by itself), and so are the counts drawn from it.
    if kind == "sample" or (kind == "sweep" and case["precision"] == "c128"):
        return "exact"
    if case.get("precision") == "c64":
        # FP32 (or split-FP16 products with FP32 sums) through every layer: 0.4-1.7e-6 measured.
        return {"rel": 8e-6, "max": 1e-4}
    # FP64 sums in another order (1e-14 measured on a job's 64 terms).
    return {"rel": 5e-14, "max": 1e-12}


# ---------------------------------------------------------------- the same in plain complex128 torch
def _matrix(op, params=None):
    """A named gate's matrix; params: its parameters (tensors for one matrix per binding)."""
    p = [torch.as_tensor(v, dtype=torch.float64, device="cuda") for v in (op[2] if params is None else params)]
    j, one = 1j, torch.ones((), dtype=torch.complex128, device="cuda")
    name = op[0]
    if name == OP["u"]:
        t, f, l = p
        c, s = torch.cos(t / 2), torch.sin(t / 2)
        return [[c * one, -torch.exp(j * l) * s], [torch.exp(j * f) * s, torch.exp(j * (f + l)) * c]]
    if name == OP["ry"]:
        c, s = torch.cos(p[0] / 2) * one, torch.sin(p[0] / 2) * one
        return [[c, -s], [s, c]]
    if name == OP["rz"]:
        return [[torch.exp(-j * p[0] / 2), 0], [0, torch.exp(j * p[0] / 2)]]
    if name == OP["h"]:
        h = math.sqrt(0.5)
        return [[h, h], [h, -h]]
    if name == OP["cz"]:
        return [[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 1, 0], [0, 0, 0, -1]]
    if name == OP["cp"]:
        return [[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 1, 0], [0, 0, 0, torch.exp(j * p[0])]]
    if name == OP["swap"]:
        return [[1, 0, 0, 0], [0, 0, 1, 0], [0, 1, 0, 0], [0, 0, 0, 1]]
    if name == OP["cx"]:  # operand 0 controls
        return [[1, 0, 0, 0], [0, 0, 0, 1], [0, 0, 1, 0], [0, 1, 0, 0]]
    raise ValueError(name)


def _evolve(psi, m, qubits):
    """m (bit i of its index is qubits[i]) on psi of shape (batch, 2^n), in place."""
    b, size = psi.shape
    order = sorted(qubits)
    shape, below = [], 0
    for q in order:
        shape = [2, 1 << (q - below)] + shape
        below = q + 1
    view = psi.view([b, size >> below] + shape)
    parts = []
    for e in range(1 << len(qubits)):
        at = [slice(None), slice(None)]
        for q in reversed(order):
            at += [(e >> qubits.index(q)) & 1, slice(None)]
        parts.append(view[tuple(at)])

    def entry(v):
        return v.reshape([-1] + [1] * (parts[0].dim() - 1)) if isinstance(v, torch.Tensor) and v.dim() else v

    new = []
    for r, row in enumerate(m):
        acc = None
        for c, v in enumerate(row):
            if isinstance(v, (int, float, complex)) and v == 0:
                continue
            t = parts[c] if isinstance(v, (int, float, complex)) and v == 1 else entry(v) * parts[c]
            acc = t if acc is None else acc + t
        same = acc is parts[r]
        new.append(None if same else torch.zeros_like(parts[r]) if acc is None else acc)
    new = [None if v is None else v.clone() if any(v is p for p in parts) else v for v in new]
    for p, v in zip(parts, new):
        if v is not None:
            p.copy_(v)


def _zero_state(n, batch=1):
    psi = torch.zeros((batch, 1 << n), dtype=torch.complex128, device="cuda")
    psi[:, 0] = 1
    return psi


def _final_state(circ):
    psi = _zero_state(circ.num_qubits)
    for op in circ.ops:
        _evolve(psi, _matrix(op), list(op[1]))
    return psi


def _signs(j, z):
    v = j & z
    for k in (32, 16, 8, 4, 2, 1):
        v = v ^ (v >> k)
    return 1.0 - 2.0 * (v & 1).double()


def _means(psi, paulis):
    """<P> for each string and row of psi: P = i^|x&z| X^x Z^z."""
    j = torch.arange(psi.shape[1], device="cuda")
    out = []
    for x, z in paulis:
        t = (psi.conj()[:, j ^ x] * (psi * _signs(j, z))).sum(1)
        out.append(1j ** (bin(x & z).count("1") % 4) * t)
    return torch.stack(out, 1)


class _Words:
    """std::mt19937_64 (Matsumoto and Nishimura's 64-bit Mersenne Twister)."""

    def __init__(self, seed):
        self.mt, self.at = [seed & (2 ** 64 - 1)], 312
        for i in range(1, 312):
            p = self.mt[-1]
            self.mt.append((6364136223846793005 * (p ^ (p >> 62)) + i) & (2 ** 64 - 1))

    def uniform(self):
        mt = self.mt
        if self.at == 312:
            for i in range(312):
                y = (mt[i] & 0xFFFFFFFF80000000) | (mt[(i + 1) % 312] & 0x7FFFFFFF)
                mt[i] = mt[(i + 156) % 312] ^ (y >> 1) ^ (0xB5026F5AA96619E9 if y & 1 else 0)
            self.at = 0
        x = mt[self.at]
        self.at += 1
        x ^= (x >> 29) & 0x5555555555555555
        x ^= (x << 17) & 0x71D67FFFEDA60000
        x ^= (x << 37) & 0xFFF7EEE000000000
        x ^= x >> 43
        return (x >> 11) * 2.0 ** -53


def _exact_trajectories(case, seed):
    n, count = case["qubits"], case["count"]
    circ = _noisy(n, case["depth"], seed)
    paulis = workloads.pauli_strings(n, case["terms"], seed + 1)
    rows = []
    for t in range(count):
        z = (seed + 2 + (t + 1) * 0x9E3779B97F4A7C15) & (2 ** 64 - 1)  # output t of SplitMix64
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & (2 ** 64 - 1)
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & (2 ** 64 - 1)
        words = _Words(z ^ (z >> 31))
        psi = _zero_state(n)
        for op in circ.ops:
            if op[0] != OP["channel"]:
                _evolve(psi, _matrix(op), list(op[1]))
                continue
            q, = op[1]
            v = psi.view(-1, 2, 1 << q)
            rho = torch.einsum("axb,ayb->xy", v, v.conj()).cpu().numpy()
            u, reached, branch = words.uniform(), 0.0, 0
            for i, k in enumerate(op[3]):
                p = float(np.trace(k.conj().T @ k @ rho).real)
                if p > 0:
                    branch, reached = i, reached + p
                    if u < reached:
                        break
            _evolve(psi, op[3][branch].tolist(), [q])
            psi /= torch.linalg.vector_norm(psi)
        rows.append(_means(psi, paulis)[0])
    rows = torch.stack(rows)
    value = rows.sum(1).real
    error = math.sqrt(float(value.var()) / count) if count > 1 else 0.0
    return {"terms": rows.mean(0).cpu().numpy(), "standard_error": error}


def exact(case, seed):
    kind = case["kind"]
    none = {"outcomes": None, "counts": None}
    if kind == "sample":
        return None  # whole numbers only
    if kind == "trajectories":
        return _exact_trajectories(case, seed)
    if kind == "serve":
        values = []
        for r in _stream(case, seed):
            values.append(0.0)
            if r["output"] != "counts":
                t = _means(_final_state(r["circuit"]), r["paulis"])[0].real.cpu().numpy()
                values[-1] = float(np.dot(t, r["coefs"]))
        return {"values": np.array(values), "sample": none}
    n = case["qubits"]
    if kind == "sweep" and n > 28:
        return None  # minutes
    circ = _circuit(case, seed)
    if kind == "bindings":
        rows = np.random.default_rng(seed).uniform(-math.pi, math.pi, (case["bindings"], 2 * n * case["layers"]))
        rows = torch.as_tensor(rows, device="cuda")
        coefs = torch.as_tensor(workloads.weights(case["terms"], seed + 2), dtype=torch.float64, device="cuda")
        out = []
        for part in rows.split(max(1, (1 << 25) >> n)):
            psi, k = _zero_state(n, len(part)), 0
            for op in circ.ops:
                _evolve(psi, _matrix(op, [part[:, k + i] for i in range(len(op[2]))]), list(op[1]))
                k += len(op[2])
            out.append((_means(psi, workloads.pauli_strings(n, case["terms"], seed + 1)).real * coefs).sum(1))
        return torch.cat(out).cpu().numpy()
    if kind == "density":
        psi = _zero_state(2 * n)
        for op in circ.ops:
            if op[0] == OP["channel"]:
                q, = op[1]
                m = sum(np.kron(k.conj(), k) for k in op[3])  # bit 0 of the index: the row qubit
                _evolve(psi, m.tolist(), [q, q + n])
            else:
                m = _matrix(op)
                qs = list(op[1])
                _evolve(psi, m, qs)
                _evolve(psi, [[v.conj() if isinstance(v, torch.Tensor) else v for v in row] for row in m],
                        [q + n for q in qs])
        rho = psi[0].view(1 << n, 1 << n).T  # entry (r, c) at r | c << n
        j = torch.arange(1 << n, device="cuda")
        terms = [1j ** (bin(x & z).count("1") % 4) * (_signs(j, z) * rho[j, j ^ x]).sum()
                 for x, z in workloads.pauli_strings(n, case["terms"], seed + 1)]
        return {"rho": torch.view_as_real(psi[0]), "terms": torch.stack(terms).cpu().numpy(), "sample": none}
    psi = _final_state(circ)
    if kind == "sweep":
        return torch.view_as_real(psi[0])
    if kind == "paulis":
        return _means(psi, workloads.pauli_strings(n, case["terms"], seed + 1))[0].cpu().numpy()
    terms = _means(psi, workloads.pauli_strings(n, case["paulis"], seed + 1))[0] if case["paulis"] else None
    return {"state": psi[0].cpu().numpy() if case["statevector"] else None,
            "terms": None if terms is None else terms.cpu().numpy(), "sample": none}
