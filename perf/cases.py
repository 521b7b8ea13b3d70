"""The performance cases of the engine: the calls a user's program makes.

Every case goes through the public entry points (``Device.execute`` on op
dicts, the layer calls and measurements of ``StateVector``, ``AdjointEnergy``
under torch.autograd, ``CircuitBatch``).  ``kind`` selects the call:

  circuit   one op-dict circuit from |0...0> to its probability vector on the
            host ("config": Haar U(2) + RZZ + CNOT ladder layers, "mixed":
            layers of many gate names)
  layer     one such layer on a resident state (a step of a deep circuit)
  qft       a QFT / inverse QFT on a register, a sub-range or ordered wires
  zz        exp(-i sum theta_b Z_a Z_b) over a graph's bonds (a QAOA cost
            layer: a chain, or a ring with a random matching)
  sample    seeded shots of all or some qubits
  marginal  the probabilities of some qubits
  expval    <P> for the words of an observable
  grad      energy and adjoint gradient of a layered ansatz
  batch     many ansatz circuits in one graph launch
"""
import math

import numpy as np
import torch

from mettleq_b200 import batch as B
from mettleq_b200 import workloads as W
from mettleq_b200.adjoint import AdjointEnergy, AdjointEngine, LayeredAnsatz, PauliSum
from mettleq_b200.device import Device
from mettleq_b200.engine import StateVector


def listed():
    return [
        # the smallest call: a short program of many gate names, as an SDK sends it
        {"name": "program-12q", "kind": "circuit", "gates": "mixed", "n": 12, "size": 4, "dtype": "complex64"},
        # the plain configuration: 20 qubits, 20 layers
        {"name": "circuit-20q", "kind": "circuit", "gates": "config", "n": 20, "size": 20, "dtype": "complex64"},
        # the scale configuration's layer, and its largest state
        {"name": "layer-30q", "kind": "layer", "n": 30, "dtype": "complex64"},
        # the same layer in double precision (the check of every complex64 result)
        {"name": "layer-25q-c128", "kind": "layer", "n": 25, "dtype": "complex128"},
        # the scale configuration's QFT layer on an odd register
        {"name": "qft-29q", "kind": "qft", "n": 29, "k": 29, "wires": "range", "inverse": False, "dtype": "complex64"},
        # phase estimation: inverse QFT on ordered wires of a larger register
        {"name": "iqft-15of25q", "kind": "qft", "n": 25, "k": 15, "wires": "ordered", "inverse": True,
         "dtype": "complex64"},
        # a QAOA cost layer on a random graph (bonds far apart)
        {"name": "zz-graph-26q", "kind": "zz", "n": 26, "graph": "random", "dtype": "complex64"},
        # 1000 shots of a large state
        {"name": "sample-28q", "kind": "sample", "n": 28, "k": 28, "shots": 1000, "dtype": "complex64"},
        # the read-out register's distribution
        {"name": "marginal-27q", "kind": "marginal", "n": 27, "k": 9, "dtype": "complex64"},
        # the energy terms of a transverse-field chain
        {"name": "expval-25q", "kind": "expval", "n": 25, "words": "ising", "count": 49, "dtype": "complex64"},
        # the differentiation configuration: 24 qubits, 8 layers, 384 parameters
        {"name": "grad-24q", "kind": "grad", "n": 24, "layers": 8, "dtype": "complex64"},
        # a batch of uneven circuits
        {"name": "batch-256", "kind": "batch", "count": 256, "lo": 10, "hi": 20, "dtype": "complex64"},
    ]


def draw(rng):
    kind = rng.choice(["circuit", "layer", "qft", "zz", "sample", "marginal", "expval", "grad", "batch"])
    dtype = rng.choice(["complex64", "complex64", "complex64", "complex128"])
    top = 27 if dtype == "complex64" else 26
    n = rng.randint(6, top)
    c = {"kind": kind, "n": n, "dtype": dtype}
    if kind == "circuit":
        gates = rng.choice(["config", "mixed"])
        c.update(n=rng.randint(5, 21), gates=gates, size=rng.randint(2, 24) if gates == "config" else rng.randint(1, 8))
    elif kind == "qft":
        c.update(k=rng.randint(2, n), wires=rng.choice(["range", "ordered"]), inverse=rng.random() < 0.5)
    elif kind == "zz":
        c.update(graph=rng.choice(["chain", "random"]))
    elif kind == "sample":
        c.update(k=rng.choice([n, rng.randint(1, n)]), shots=int(round(10 ** rng.uniform(0, 4.7))))
    elif kind == "marginal":
        c.update(k=rng.randint(1, min(n, 16)))
    elif kind == "expval":
        words = rng.choice(["ising", "heisenberg", "random"])
        c.update(n=rng.randint(6, min(top, 25)), words=words)
        c["count"] = {"ising": 2 * c["n"] - 1, "heisenberg": 3 * (c["n"] - 1), "random": rng.randint(1, 40)}[words]
    elif kind == "grad":
        c.update(n=rng.randint(4, 24 if dtype == "complex64" else 22), layers=rng.randint(1, 8))
    elif kind == "batch":
        lo = rng.randint(3, 14)
        c = {"kind": kind, "dtype": "complex64", "count": int(round(10 ** rng.uniform(0.5, 2.4))), "lo": lo,
             "hi": min(20, lo + rng.randint(0, 8))}
    return c


# ------------------------------------------------------------------ inputs
class _Memory:
    """A resident state for torch.as_tensor (real and imaginary parts
    interleaved); the tensor keeps it, and so the state, alive."""

    def __init__(self, sv):
        self.sv = sv
        self.__cuda_array_interface__ = {"data": (sv.device_ptr(), False), "shape": (2 << sv.n,), "version": 2,
                                         "typestr": "<f4" if sv.dtype == np.complex64 else "<f8"}


def _view(sv):
    """The resident amplitudes as a flat torch tensor of reals (no copy)."""
    return torch.as_tensor(_Memory(sv), device="cuda")


def _fill(v, n, seed):
    """A random state, as random circuits leave it."""
    v.normal_(0.0, math.sqrt(0.5 / (1 << n)), generator=torch.Generator(device="cuda").manual_seed(seed))
    v.div_(torch.linalg.vector_norm(v, dtype=torch.float64).to(v.dtype))


def _state(n, dtype, seed):
    """The same state in 64 bits, as a plain torch tensor."""
    v = torch.empty(2 << n, dtype=torch.float32 if dtype == "complex64" else torch.float64, device="cuda")
    _fill(v, n, seed)
    return torch.view_as_complex(v.double().view(-1, 2))


def _inputs(c, seed):
    """The call's host-side arguments, from the seed alone."""
    kind, n = c["kind"], c.get("n", 0)
    rng = np.random.default_rng([seed, 7])
    if kind == "circuit":
        if c["gates"] == "config":
            return {"ops": W.plain_circuit(n, c["size"], seed).ops()[0]}
        return {"ops": _program(n, c["size"], rng)}
    if kind == "layer":
        return {"mats": np.stack([W.haar_u2(rng).reshape(4) for _ in range(n)]),
                "terms": [(0, i, i + 1, [float(t) / 2.0]) for i, t in enumerate(rng.uniform(0.0, 2.0 * math.pi, n - 1))]}
    if kind == "qft":
        if c["wires"] == "range":
            q0 = int(rng.integers(0, n - c["k"] + 1))
            return {"wires": list(range(q0, q0 + c["k"]))}
        return {"wires": [int(w) for w in rng.permutation(n)[:c["k"]]]}
    if kind == "zz":
        bonds = [(i, i + 1) for i in range(n - 1)]
        if c["graph"] == "random":  # a ring and a random perfect matching
            m = [int(w) for w in rng.permutation(n)]
            bonds = sorted({tuple(sorted(e)) for e in bonds + [(n - 1, 0)] + list(zip(m[0::2], m[1::2]))})
        return {"bonds": bonds, "thetas": [float(t) for t in rng.uniform(0.0, math.pi, len(bonds))]}
    if kind in ("sample", "marginal"):
        k = c["k"]
        return {"wires": None if k == n else [int(w) for w in rng.permutation(n)[:k]], "seed": int(rng.integers(1 << 32))}
    if kind == "expval":
        if c["words"] == "ising":
            words = [{i: "Z", i + 1: "Z"} for i in range(n - 1)] + [{i: "X"} for i in range(n)]
        elif c["words"] == "heisenberg":
            words = [{i: p, i + 1: p} for p in "XYZ" for i in range(n - 1)]
        else:
            words = [{int(w): "XYZ"[int(rng.integers(3))] for w in rng.permutation(n)[:int(rng.integers(1, min(n, 6) + 1))]}
                     for _ in range(c["count"])]
        return {"words": words}
    if kind == "grad":
        return {"params": rng.uniform(-math.pi, math.pi, (c["layers"], n, 2))}
    ns, depths, params = B.hea_batch(c["count"], c["count"], (c["lo"], c["hi"]), (4, 16))
    return {"ns": ns, "depths": depths, "mats": [B.hea_mats(rng.uniform(-math.pi, math.pi, p.shape)) for p in params]}


def _program(n, layers, rng):
    """Layers of a random one-qubit gate on every wire and a chain of one
    random two-qubit gate."""
    one = {"H": 0, "Y": 0, "SX": 0, "RX": 1, "RY": 1, "U3": 3, "S": 0, "T": 0, "RZ": 1, "U1": 1}
    two = {"CNOT": 0, "CZ": 0, "CPHASE": 1, "CRX": 1, "CRY": 1, "CRZ": 1, "CH": 0, "SWAP": 0, "XXPHASE": 1, "YYPHASE": 1,
           "ZZPHASE": 1}

    def op(name, wires, count):
        return {"name": name, "wires": wires, "parameters": [float(x) for x in rng.uniform(-math.pi, math.pi, count)]}

    ops = []
    for _ in range(layers):
        for q in range(n):
            name = list(one)[int(rng.integers(len(one)))]
            ops.append(op(name, [q], one[name]))
        name = list(two)[int(rng.integers(len(two)))]
        ops += [op(name, [q, q + 1], two[name]) for q in range(n - 1)]
    return ops


# ------------------------------------------------------------------ the calls
def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c, **_inputs(c, seed)}
    if kind == "circuit":
        s["device"] = Device(c["n"], dtype=c["dtype"])
    elif kind == "grad":
        s["stream"] = torch.cuda.Stream()  # both of the engine's states run on the program's stream
        s["engine"] = AdjointEngine(LayeredAnsatz(c["n"], c["layers"]), PauliSum.ising_chain(c["n"]), dtype=c["dtype"],
                                    stream=s["stream"].cuda_stream)
        s["p"] = torch.tensor(s["params"], requires_grad=True)
    elif kind == "batch":
        s["batch"] = B.CircuitBatch(s["ns"], s["depths"], lanes=16)
        s["packed"] = s["batch"].pack(s["mats"])
    else:
        s["sv"] = StateVector(c["n"], dtype=c["dtype"])
        s["sv"].synchronize()
        _fill(_view(s["sv"]), c["n"], seed)
        if kind == "layer":
            s["rows"], s["c"] = W.cnot_ladder_rows(c["n"])
    torch.cuda.synchronize()
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "circuit":
        s["device"].reset()
        return s["device"].execute(s["ops"]).probabilities_array()
    if kind == "grad":
        s["p"].grad = None
        e = AdjointEnergy.apply(s["p"], s["engine"])
        e.backward()
        return [e.detach(), s["p"].grad]
    if kind == "batch":
        s["batch"].run(packed=s["packed"])
        return [s["batch"].z0(), s["batch"].probs_dev]
    sv = s["sv"]
    if kind == "sample":
        return sv.sample_indices(c["shots"], s["wires"], seed=s["seed"])
    if kind == "marginal":
        return sv.probabilities(s["wires"] if s["wires"] is not None else list(range(c["n"])))
    if kind == "expval":
        return sv.expval_pauli(s["words"])
    if kind == "layer":
        sv.apply_layer(s["mats"], None, s["terms"], s["rows"], s["c"])
    elif kind == "qft":
        sv.apply_qft(s["wires"], c["inverse"])
    else:
        sv.apply_zz_weighted(s["bonds"], s["thetas"])
    return _view(sv)


def work(case):
    c, kind = case, case["kind"]
    dim = float(1 << c.get("n", 0))
    state = dim * (8 if c["dtype"] == "complex64" else 16)
    n = c.get("n", 0)
    if kind == "circuit":
        gates = c["size"] * (3 * n - 2 if c["gates"] == "config" else 2 * n - 1)
        return {"bytes": 4 * dim + 64 * gates, "flops": 8 * dim * gates}
    if kind == "layer":
        return {"bytes": 2 * state, "flops": dim * (14 * n + 6)}
    if kind == "qft":
        return {"bytes": 2 * state, "flops": dim * 7 * c["k"]}
    if kind == "zz":
        return {"bytes": 2 * state, "flops": 6 * dim}
    if kind == "sample":
        return {"bytes": state + 8 * c["shots"], "flops": 4 * dim}
    if kind == "marginal":
        return {"bytes": state + 8 * 2.0 ** c["k"], "flops": 4 * dim}
    if kind == "expval":
        return {"bytes": state, "flops": 8 * dim * c["count"]}
    if kind == "grad":
        # psi and lambda: written by the forward part, read and written once per layer backward
        return {"bytes": 4 * state * c["layers"], "flops": dim * c["layers"] * n * (14 + 2 * 14 + 24)}
    ns, depths, _ = B.hea_batch(c["count"], c["count"], (c["lo"], c["hi"]), (4, 16))
    return {"bytes": sum(4.0 * 2.0 ** m + 64.0 * m * d for m, d in zip(ns, depths)),
            "flops": sum(14.0 * m * d * 2.0 ** m for m, d in zip(ns, depths))}


# ------------------------------------------------------------------ 64 bits
def _gate(x, n, q, u):
    """A 2x2 on qubit q (index bit n-1-q) of the complex128 state x, in place."""
    v = x.view(1 << q, 2, -1)
    a, b = v[:, 0].clone(), v[:, 1]
    u = [complex(t) for t in np.asarray(u, dtype=np.complex128).reshape(4)]
    v[:, 0] = a * u[0] + b * u[1]
    v[:, 1] = a * u[2] + b * u[3]


def _pair(x, n, a, b, d):
    """diag(d) on qubits (a, b)."""
    t = torch.tensor(np.asarray(d, dtype=np.complex128).reshape(2, 2), device="cuda")
    if a > b:
        a, b, t = b, a, t.t()
    x.view(1 << a, 2, 1 << (b - a - 1), 2, -1).mul_(t.reshape(1, 2, 1, 2, 1))


def _ladder(x, n):
    """CNOT(0, 1), ..., CNOT(n-2, n-1)."""
    i = torch.arange(1 << n, device="cuda", dtype=torch.int64)
    return x[i ^ (i >> 1)]


_SQ = math.sqrt(0.5)
_FIXED = {"H": [_SQ, _SQ, _SQ, -_SQ], "X": [0, 1, 1, 0], "Y": [0, -1j, 1j, 0], "Z": [1, 0, 0, -1], "S": [1, 0, 0, 1j],
          "T": [1, 0, 0, _SQ + _SQ * 1j], "SX": [0.5 + 0.5j, 0.5 - 0.5j, 0.5 - 0.5j, 0.5 + 0.5j]}


def _matrix(name, p):
    if name in _FIXED:
        return np.array(_FIXED[name], dtype=np.complex128).reshape(2, 2)
    t = p[0]
    c, s = math.cos(t / 2), math.sin(t / 2)
    if name == "RX":
        return np.array([[c, -1j * s], [-1j * s, c]])
    if name == "RY":
        return np.array([[c, -s], [s, c]], dtype=np.complex128)
    if name == "RZ":
        return np.diag(np.exp([-0.5j * t, 0.5j * t]))
    if name == "U1":
        return np.diag([1, np.exp(1j * t)])
    return _matrix("RZ", [p[1]]) @ _matrix("RY", [p[0]]) @ _matrix("RZ", [p[2]])  # U3


def _dense(x, n, wires, m):
    """A dense matrix on the listed wires (first = most significant)."""
    k = len(wires)
    order = list(wires) + [q for q in range(n) if q not in wires]
    v = x.view([2] * n).permute(order).reshape(1 << k, -1)
    v = torch.tensor(np.asarray(m, dtype=np.complex128), device="cuda") @ v
    back = [0] * n
    for i, q in enumerate(order):
        back[q] = i
    return v.view([2] * n).permute(back).reshape(-1).contiguous()


def _op(x, n, op):
    name, w, p = op["name"], op["wires"], op["parameters"]
    if len(w) == 1:
        _gate(x, n, w[0], _matrix(name, p))
        return x
    if name in ("ZZPHASE", "CZ", "CPHASE", "CRZ"):
        t = p[0] if p else math.pi
        e = {"ZZPHASE": [-t, t, t, -t], "CZ": [0, 0, 0, t], "CPHASE": [0, 0, 0, t], "CRZ": [0, 0, -t / 2, t / 2]}[name]
        _pair(x, n, w[0], w[1], np.exp(1j * np.array(e)))
        return x
    if name in ("XXPHASE", "YYPHASE"):
        m = np.kron(*[_matrix(name[0], p)] * 2)
        m = math.cos(p[0]) * np.eye(4) - 1j * math.sin(p[0]) * m
    elif name == "SWAP":
        m = np.eye(4)[[0, 2, 1, 3]]
    else:
        m = np.eye(4, dtype=np.complex128)
        m[2:, 2:] = _matrix({"CNOT": "X", "CH": "H", "CRX": "RX", "CRY": "RY"}[name], p)
    return _dense(x, n, w, m)


def _zero(n):
    x = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    x[0] = 1
    return x


def _word(x, n, word):
    """P x for a Pauli word."""
    y = x.clone()
    for q, p in word.items():
        _gate(y, n, q, _FIXED[p])
    return y


def _exact_grad(c, s):
    n, p = c["n"], s["params"]
    mats = [[_matrix("RZ", [p[l, q, 1]]) @ _matrix("RY", [p[l, q, 0]]) for q in range(n)] for l in range(c["layers"])]
    x = _zero(n)
    for l in range(c["layers"]):
        for q in range(n):
            _gate(x, n, q, mats[l][q])
        x = _ladder(x, n)
    y = torch.zeros_like(x)
    for word, coef in PauliSum.ising_chain(n).words():
        y += coef * _word(x, n, word)
    energy = torch.vdot(x, y).real
    grad = np.zeros(p.shape)
    i = torch.arange(1 << n, device="cuda", dtype=torch.int64)
    back = torch.empty_like(i)
    back[i ^ (i >> 1)] = i
    for l in reversed(range(c["layers"])):
        x, y = x[back], y[back]
        for q in range(n):
            for k, name in ((1, "Z"), (0, "Y")):
                z = x.clone()
                _gate(z, n, q, _FIXED[name])
                grad[l, q, k] = float(torch.vdot(y, z).imag)
                u = _matrix("R" + name, [p[l, q, k]]).conj().T
                _gate(x, n, q, u)
                _gate(y, n, q, u)
    return [energy, torch.tensor(grad)]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "sample":
        return None
    s = _inputs(c, seed)
    if kind == "circuit":
        x = _zero(c["n"])
        for op in s["ops"]:
            x = _op(x, c["n"], op)
        return x.abs().square().cpu().numpy().astype(np.float64)
    if kind == "grad":
        return _exact_grad(c, s)
    if kind == "batch":
        z, probs = [], []
        for n, mats in zip(s["ns"], s["mats"]):
            x = _zero(n)
            for layer in mats:
                for q in range(n):
                    _gate(x, n, q, layer[q])
                x = _ladder(x, n)
            p = x.abs().square()
            z.append(float(p[: p.numel() // 2].sum() - p[p.numel() // 2:].sum()))
            probs.append(p)
        return [np.array(z), torch.cat(probs)]
    n = c["n"]
    x = _state(n, c["dtype"], seed)
    if kind == "marginal":
        wires = s["wires"] if s["wires"] is not None else list(range(n))
        i = torch.arange(1 << n, device="cuda", dtype=torch.int64)
        at = torch.zeros_like(i)
        for w in wires:
            at = 2 * at + ((i >> (n - 1 - w)) & 1)
        return torch.zeros(1 << len(wires), dtype=torch.float64, device="cuda").index_add_(
            0, at, torch.view_as_real(x).square().sum(1)).cpu().numpy()
    if kind == "expval":
        return np.array([complex(torch.vdot(x, _word(x, n, w))) for w in s["words"]])
    if kind == "layer":
        for q in range(n):
            _gate(x, n, q, s["mats"][q])
        for _, a, b, (t,) in s["terms"]:
            _pair(x, n, a, b, np.exp(1j * np.array([-t, t, t, -t])))
        x = _ladder(x, n)
    elif kind == "zz":
        for (a, b), t in zip(s["bonds"], s["thetas"]):
            _pair(x, n, a, b, np.exp(1j * np.array([-t, t, t, -t])))
    else:
        w, k = s["wires"], c["k"]
        stages = list(range(k))
        for j in reversed(stages) if c["inverse"] else stages:
            if not c["inverse"]:
                _gate(x, n, w[j], _FIXED["H"])
            sign = -1.0 if c["inverse"] else 1.0
            for i in range(j + 1, k):
                _pair(x, n, w[j], w[i], [1, 1, 1, np.exp(1j * sign * math.pi / 2.0 ** (i - j))])
            if c["inverse"]:
                _gate(x, n, w[j], _FIXED["H"])
    return torch.view_as_real(x).reshape(-1)
