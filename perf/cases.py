"""Performance cases of the engine: what programs have it do, over its range of sizes.

Each case is a plain dict with a ``family`` and its sizes.  ``prepare`` builds what a
program holds before the call (circuits as ``model_dump_json()`` objects, decoded batch
programs, parameter vectors), ``run`` makes one pass through the public API, ``work`` is the
path's own minimum of bytes and operations, and ``exact`` recomputes the floating outputs
in 64 bits with torch and numpy alone.

Families
  dynamic     one run of a mixed-gate circuit with measurements, conditionals and resets
  brickwork   one run of layers of u3 and cx on brickwork pairs
  qft         one run of the quantum Fourier transform of a basis state
  shots       ``simulate_shots`` of a circuit with feed-forward
  ragged      independent circuits of uneven size in one batch, with their final states
  gradient    adjoint gradient of one parameter set
  gradients   a batch of parameter sets through the torch autograd function
  mps         one matrix-product-state run
  mps_shots   shots of the feed-forward circuit on matrix-product states
"""
import json
import math

import numpy as np
import torch

from dqsim_bosonic_b200 import MpsSimulator, StatevectorSimulator
from dqsim_bosonic_b200.adjoint import Param, ParamCircuit, PauliSum, adjoint_gradient, expval
from dqsim_bosonic_b200.batch import run_batch
from dqsim_bosonic_b200.circuit import decode_program


def listed():
    return [
        # a teleportation-sized dynamic circuit, run interactively: latency alone
        {"name": "dynamic5", "family": "dynamic", "n": 5, "gates": 30, "groups": 3, "exec": "fused", "seen": "host"},
        # a ten-qubit-or-less benchmark circuit with the API's default number of shots
        {"name": "shots7", "family": "shots", "n": 7, "layers": 6, "shots": 1000},
        # the plain 20-qubit workload: final state on the host and 10000 samples
        {"name": "brickwork20", "family": "brickwork", "n": 20, "layers": 20, "seen": "host"},
        # exact arithmetic gate by gate on an ordinary state, with feed-forward
        {"name": "dynamic22", "family": "dynamic", "n": 22, "gates": 120, "groups": 4, "exec": "per_gate", "seen": "device"},
        # a deep circuit on a state far larger than the caches
        {"name": "brickwork28", "family": "brickwork", "n": 28, "layers": 20, "seen": "device"},
        # the 30-qubit Fourier transform: marginals of ten qubits and the state in place
        {"name": "qft30", "family": "qft", "n": 30, "seen": "device"},
        # 4096 shots of a 16-qubit circuit with mid-circuit measurement
        {"name": "shots16", "family": "shots", "n": 16, "layers": 12, "shots": 4096},
        # circuits of 10 to 20 qubits and 5 to 40 layers in one batch
        {"name": "ragged48", "family": "ragged", "items": 48, "n_lo": 10, "n_hi": 20, "d_lo": 5, "d_hi": 40},
        # gradient of a 24-qubit, 1152-parameter ansatz
        {"name": "gradient24", "family": "gradient", "n": 24, "layers": 16},
        # one optimiser step's gradients of 128 sets of a 20-qubit ansatz
        {"name": "gradients20", "family": "gradients", "n": 20, "layers": 8, "sets": 128},
        # 4096 shots of the same feed-forward circuit on matrix-product states
        {"name": "mps_shots16", "family": "mps_shots", "n": 16, "layers": 12, "shots": 4096, "bond": 16},
        # one truncated matrix-product-state run
        {"name": "mps20", "family": "mps", "n": 20, "layers": 20, "bond": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["dynamic", "brickwork", "qft", "shots", "ragged", "gradient", "gradients", "mps", "mps_shots"])
    if family == "dynamic":
        n = rng.randint(3, 23)
        return {"family": family, "n": n, "gates": _log(rng, 20, 150), "groups": rng.randint(1, 5),
                "exec": rng.choice(["fused", "fused", "per_gate"]), "seen": "host" if n < 20 else "device"}
    if family == "brickwork":
        n = rng.randint(6, 28)
        return {"family": family, "n": n, "layers": _log(rng, 3, 20), "seen": "host" if n <= 20 else "device"}
    if family == "qft":
        n = rng.randint(6, 30)
        return {"family": family, "n": n, "seen": "host" if n <= 20 else "device"}
    if family == "shots":
        return {"family": family, "n": rng.randint(3, 16), "layers": rng.randint(3, 12), "shots": _log(rng, 100, 4096)}
    if family == "ragged":
        return {"family": family, "items": _log(rng, 6, 60), "n_lo": 10, "n_hi": rng.randint(12, 21),
                "d_lo": 5, "d_hi": rng.randint(8, 40)}
    if family == "gradient":
        return {"family": family, "n": rng.randint(6, 25), "layers": rng.randint(1, 12)}
    if family == "gradients":
        n = rng.randint(8, 20)
        return {"family": family, "n": n, "layers": rng.randint(1, 8), "sets": _log(rng, 4, 128)}
    if family == "mps":
        return {"family": family, "n": rng.randint(6, 21), "layers": rng.randint(4, 20), "bond": _log(rng, 6, 64)}
    return {"family": family, "n": rng.randint(4, 16), "layers": rng.randint(3, 12), "shots": _log(rng, 100, 4096),
            "bond": rng.randint(4, 16)}


# ---- circuits -------------------------------------------------------------------------

_FIELDS = {
    "h": ("qubit",), "x": ("qubit",), "t": ("qubit",), "sx": ("qubit",), "reset": ("qubit",),
    "rx": ("qubit", "theta"), "rz": ("qubit", "phi"), "u3": ("qubit", "theta", "phi", "lam"),
    "cx": ("control", "target"), "cz": ("control", "target"), "swap": ("a", "b"),
    "cp": ("control", "target", "lam"), "rxx": ("a", "b", "theta"), "rzz": ("a", "b", "theta"),
    "ccx": ("control1", "control2", "target"), "measure": ("qubit", "cbit"),
}
_ARITY = {"h": 1, "x": 1, "t": 1, "sx": 1, "rx": 1, "rz": 1, "u3": 1, "reset": 1, "measure": 1,
          "cx": 2, "cz": 2, "swap": 2, "cp": 2, "rxx": 2, "rzz": 2, "ccx": 3}
_MIXED = ["u3", "u3", "h", "t", "sx", "rx", "rz", "cx", "cx", "cz", "swap", "cp", "rxx", "rzz", "ccx"]


class Circuit:
    """A circuit model: its instructions (kind, qubits, values[, condition]) and JSON dump."""

    def __init__(self, n, ops, ncbits=0):
        self.n, self.ops, self.ncbits = n, ops, ncbits
        insts = []
        for kind, qs, vals, cnd in ops:
            d = dict(zip(_FIELDS[kind], list(qs) + list(vals)), kind=kind, qubits=list(qs),
                     params=[] if kind == "measure" else list(vals))
            if cnd is not None:
                d = {"kind": "conditional", "op": d, "qubits": list(qs),
                     "condition": {"creg_base": cnd[0], "creg_size": 1, "creg_value": cnd[1]}}
            insts.append(d)
        cregs = {"c": {"name": "c", "size": ncbits, "base": 0}} if ncbits else {}
        self.text = json.dumps({"qregs": {"q": {"name": "q", "size": n, "base": 0}}, "cregs": cregs,
                                "instructions": insts})

    def model_dump_json(self):
        return self.text


def _layer(rng, n, k, ops):
    ang = rng.uniform(0.0, 2.0 * math.pi, size=(n, 3))
    ops += [("u3", (q,), ang[q].tolist(), None) for q in range(n)]
    ops += [("cx", (q, q + 1), (), None) for q in range(k % 2, n - 1, 2)]


def _brickwork(n, layers, rng):
    ops = []
    for k in range(layers):
        _layer(rng, n, k, ops)
    return Circuit(n, ops)


def _qft(n, rng):
    bits = rng.random(n) < 0.5
    ops = [("x", (q,), (), None) for q in range(n) if bits[q]]
    for j in range(n):
        ops.append(("h", (j,), (), None))
        ops += [("cp", (k, j), (math.pi / 2 ** (k - j),), None) for k in range(j + 1, n)]
    ops += [("swap", (j, n - 1 - j), (), None) for j in range(n // 2)]
    return Circuit(n, ops), sum(1 << q for q in range(n) if bits[q])


def _dynamic(case, rng):
    n, groups = case["n"], case["groups"]
    per = max(1, case["gates"] // (groups + 1))
    ops = []
    for k in range(groups + 1):
        for _ in range(per):
            kind = _MIXED[rng.integers(len(_MIXED))]
            qs = rng.permutation(n)[: _ARITY[kind]].tolist()
            nv = len(_FIELDS[kind]) - len(qs)
            ops.append((kind, tuple(qs), rng.uniform(0, 2 * math.pi, nv).tolist(), None))
        if k < groups:
            a, b, c = rng.permutation(n)[:3].tolist()
            ops += [("measure", (a,), (k,), None), ("x", (b,), (), (k, 1)), ("reset", (c,), (), None)]
    return Circuit(n, ops, groups)


def _feed_forward(case, rng):
    """u3 + cx layers; every third one measures qubit 0 into a bit of its own, flips qubit 1
    on it and resets qubit 0.  Up to ten qubits, a last measurement of every qubit."""
    n, layers = case["n"], case["layers"]
    ops, c = [], 0
    for k in range(layers):
        _layer(rng, n, k, ops)
        if k % 3 == 2:
            ops += [("measure", (0,), (c,), None), ("x", (1,), (), (c, 1)), ("reset", (0,), (), None)]
            c += 1
    if n <= 10:
        ops += [("measure", (q,), (c + q,), None) for q in range(n)]
        c += n
    return Circuit(n, ops, c)


def _ansatz(n, layers):
    c = ParamCircuit(n)
    k = 0
    for _ in range(layers):
        for q in range(n):
            c.ry(q, Param(k + q))
        for q in range(n):
            c.rz(q, Param(k + n + q))
        for q in range(n):
            c.rzz(q, (q + 1) % n, Param(k + 2 * n + q))
        k += 3 * n
    return c


def _observable(n, seed):
    rng = np.random.default_rng(seed + 5)
    a, b = rng.normal(size=n), rng.normal(size=n)
    terms = [(float(a[i]), {i: "Z", (i + 1) % n: "Z"}) for i in range(n)]
    return a, b, PauliSum(terms + [(float(b[i]), {i: "X"}) for i in range(n)])


def _theta(case, seed):
    shape = (case.get("sets", 1), case["layers"] * 3 * case["n"])
    return np.random.default_rng(seed).uniform(-math.pi, math.pi, size=shape)


def _ragged(case, rng):
    """Sizes over the range in a fixed spread (the same for every seed), angles by the seed."""
    k, got = case["items"], []
    for i in range(k):
        n = case["n_lo"] + i * (case["n_hi"] - case["n_lo"] + 1) // k
        d = case["d_lo"] + (i * 7919 % k) * (case["d_hi"] - case["d_lo"] + 1) // k
        got.append(_brickwork(n, d, rng))
    return got


# ---- one pass -------------------------------------------------------------------------


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    f, s = case["family"], {"case": case, "seed": seed}
    if f == "dynamic":
        s["circuit"] = _dynamic(case, rng)
        s["sim"] = StatevectorSimulator(seed=seed, exec=case["exec"])
    elif f == "brickwork":
        s["circuit"] = _brickwork(case["n"], case["layers"], rng)
        s["sim"] = StatevectorSimulator(seed=seed)
    elif f == "qft":
        s["circuit"], _ = _qft(case["n"], rng)
        s["sim"] = StatevectorSimulator(seed=seed)
    elif f == "shots":
        s["circuit"] = _feed_forward(case, rng)
        s["sim"] = StatevectorSimulator(seed=seed)
    elif f == "ragged":
        s["programs"] = [decode_program(c.model_dump_json()) for c in _ragged(case, rng)]
        s["seeds"] = [seed + i for i in range(case["items"])]
    elif f in ("gradient", "gradients"):
        s["circuit"] = _ansatz(case["n"], case["layers"])
        s["observable"] = _observable(case["n"], seed)[2]
        th = _theta(case, seed)
        s["theta"] = th[0] if f == "gradient" else torch.tensor(th, device="cuda")
    elif f == "mps":
        s["circuit"] = _brickwork(case["n"], case["layers"], rng)
        s["sim"] = MpsSimulator(seed=seed, max_bond_dimension=case["bond"])
    else:
        s["circuit"] = _feed_forward(case, rng)
        s["sim"] = MpsSimulator(seed=seed, max_bond_dimension=case["bond"])
    return s


class _InPlace:
    """The device-resident state as a zero-copy tensor source (it keeps the state alive)."""

    def __init__(self, state):
        self.state = state
        self.__cuda_array_interface__ = {"shape": (1 << state.n,), "typestr": "<c16", "strides": None,
                                         "data": (state.device_ptr()[0], False), "version": 2}


def _state(case, result):
    if case.get("seen", "device") == "host":
        return result.statevector
    return torch.as_tensor(_InPlace(result.state_handle), device="cuda")


def _outcomes(counts):
    """Every shot's bitstring as a row of characters, in the order of their values."""
    keys = sorted(counts)
    rows = np.frombuffer("".join(keys).encode(), dtype=np.uint8).reshape(len(keys), -1)
    return np.repeat(rows, [counts[k] for k in keys], axis=0)


def run(state):
    case, f = state["case"], state["case"]["family"]
    if f == "dynamic":
        r = state["sim"].simulate(state["circuit"])
        bits = r.classical_bits
        return {"bits": np.array([bits[i] for i in range(case["groups"])], dtype=np.int64),
                "counts": _outcomes(r.counts(1000, seed=7)), "state": _state(case, r)}
    if f == "brickwork":
        r = state["sim"].simulate(state["circuit"])
        return {"counts": _outcomes(r.counts(10000, seed=7)) if case["n"] <= 20 else None, "state": _state(case, r)}
    if f == "qft":
        n = case["n"]
        r = state["sim"].simulate(state["circuit"])
        top = r.probability_array(list(range(n - 1, n - 1 - min(10, n), -1)))
        return {"top": top, "state": _state(case, r)}
    if f in ("shots", "mps_shots"):
        return _outcomes(state["sim"].simulate_shots(state["circuit"], case["shots"]))
    if f == "ragged":
        return run_batch(state["programs"], state["seeds"], want_states=True)[1]
    if f == "gradient":
        e, g = adjoint_gradient(state["circuit"], state["theta"], state["observable"])
        return {"energy": e, "gradient": g}
    if f == "gradients":
        th = state["theta"].detach().requires_grad_(True)
        e = expval(th, state["circuit"], state["observable"])
        e.sum().backward()
        return {"energy": e.detach(), "gradient": th.grad}
    return {"state": _state(case, state["sim"].simulate(state["circuit"]))}


# ---- the work a pass cannot do without --------------------------------------------------

# floating operations per amplitude of the state (a complex multiply-add pair counts 8)
_OPS = {"u3": 14, "h": 4, "sx": 8, "rx": 8, "rz": 6, "t": 3, "cp": 1.5, "rxx": 8, "rzz": 6, "measure": 2, "reset": 2}


def _gate_flops(ops, n):
    return sum(_OPS.get(o[0], 0) for o in ops) * float(1 << n)


def work(case):
    f, n = case["family"], case.get("n", 0)
    rng = np.random.default_rng(0)
    if f in ("dynamic", "brickwork", "qft"):
        c = _dynamic(case, rng) if f == "dynamic" else _brickwork(n, case["layers"], rng) if f == "brickwork" else _qft(n, rng)[0]
        return {"bytes": len(c.text) + 16.0 * (1 << n), "flops": _gate_flops(c.ops, n)}
    if f == "shots":
        c = _feed_forward(case, rng)
        return {"bytes": len(c.text) + 16.0 * case["shots"], "flops": case["shots"] * _gate_flops(c.ops, n)}
    if f == "ragged":
        cs = _ragged(case, rng)
        return {"bytes": sum(16.0 * (1 << c.n) for c in cs), "flops": sum(_gate_flops(c.ops, c.n) for c in cs)}
    if f in ("gradient", "gradients"):
        # forward, then psi and lambda back: ry 8, one combined phase per layer 6 + 6; a product per layer and kind
        sets = case.get("sets", 1)
        ops = case["layers"] * (3 * (n * 4 + 6 + 6) + 2 * (n * 2 + 6))
        return {"bytes": sets * (48.0 * n * case["layers"] + 8), "flops": sets * ops * float(1 << n)}
    # a contraction and one two-sided factorisation per step at the bond each step can reach
    steps = 0.0
    for k in range(case["layers"]):
        for q in range(k % 2, n - 1, 2):
            l, m, r = (min(2.0 ** min(j, n - j), 2.0 ** k, case["bond"]) for j in (q, q + 1, q + 2))
            rows, cols = 2 * max(l, r), 2 * min(l, r)
            steps += 32 * l * m * r + 64 * l * r + 8 * (4 * rows * cols ** 2 + 8 * cols ** 3)
    if f == "mps":
        return {"bytes": 16.0 * (1 << n), "flops": steps + 8.0 * case["bond"] * (1 << n)}
    return {"bytes": 16.0 * case["shots"], "flops": steps * case["shots"]}


# ---- the same in 64 bits, without the engine ---------------------------------------------


def _matrix(kind, v):
    i = 1j
    if kind == "h":
        return np.array([[1, 1], [1, -1]]) / math.sqrt(2)
    if kind == "x":
        return np.array([[0, 1], [1, 0]])
    if kind == "t":
        return np.diag([1, np.exp(i * math.pi / 4)])
    if kind == "sx":
        return np.array([[1 + i, 1 - i], [1 - i, 1 + i]]) / 2
    if kind == "rz":
        return np.diag([np.exp(-i * v[0] / 2), np.exp(i * v[0] / 2)])
    if kind == "rx":
        c, s = math.cos(v[0] / 2), math.sin(v[0] / 2)
        return np.array([[c, -i * s], [-i * s, c]])
    if kind == "u3":
        c, s = math.cos(v[0] / 2), math.sin(v[0] / 2)
        return np.array([[c, -np.exp(i * v[2]) * s], [np.exp(i * v[1]) * s, np.exp(i * (v[1] + v[2])) * c]])
    if kind == "cx":
        return np.eye(4)[[0, 1, 3, 2]]
    if kind == "cz":
        return np.diag([1, 1, 1, -1])
    if kind == "swap":
        return np.eye(4)[[0, 2, 1, 3]]
    if kind == "cp":
        return np.diag([1, 1, 1, np.exp(i * v[0])])
    if kind == "rzz":
        return np.diag(np.exp(-0.5j * v[0] * np.array([1, -1, -1, 1])))
    if kind == "rxx":
        return math.cos(v[0] / 2) * np.eye(4) - i * math.sin(v[0] / 2) * np.eye(4)[::-1]
    if kind == "ccx":
        return np.eye(8)[[0, 1, 2, 3, 4, 5, 7, 6]]
    raise ValueError(kind)


def _slices(psi, qs):
    """Views of `psi` for each value of the qubits `qs` (qs[0] the most significant bit)."""
    order = sorted(qs, reverse=True)
    shape, hi = [], psi.numel().bit_length() - 1
    for q in order:
        shape += [1 << (hi - q - 1), 2]
        hi = q
    v = psi.view(shape + [1 << hi])
    got = []
    for j in range(1 << len(qs)):
        at = [slice(None)] * v.dim()
        for pos, q in enumerate(order):
            at[2 * pos + 1] = (j >> (len(qs) - 1 - qs.index(q))) & 1
        got.append(v[tuple(at)])
    return got


def _apply(psi, kind, qs, vals):
    m = _matrix(kind, vals)
    parts = _slices(psi, list(qs))
    rows = [j for j in range(len(parts)) if not (m[j, j] == 1 and np.count_nonzero(m[j]) == 1)]
    new = []
    for j in rows:
        acc = None
        for k in np.flatnonzero(m[j]):
            c = complex(m[j, k])
            acc = parts[k] * c if acc is None else acc.add_(parts[k], alpha=c)
        new.append(acc)
    for j, x in zip(rows, new):
        parts[j].copy_(x)


def _zero_state(n):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1
    return psi


def _unitary(circuit):
    psi = _zero_state(circuit.n)
    for kind, qs, vals, _ in circuit.ops:
        _apply(psi, kind, qs, vals)
    return psi


def _draws(seed, count):
    """The outcome stream: ChaCha with 8 rounds (RFC 8439's block function, 64-bit counter) on
    a key of eight PCG32 (XSH-RR) outputs; a draw is 53 bits of two consecutive words."""
    m64, m32 = (1 << 64) - 1, (1 << 32) - 1
    key, s = [], seed & m64
    for _ in range(8):
        s = (s * 6364136223846793005 + 11634580027462260723) & m64
        xs, rot = (((s >> 18) ^ s) >> 27) & m32, s >> 59
        key.append(((xs >> rot) | (xs << (-rot & 31))) & m32)
    words, block = [], 0
    while len(words) < 2 * count:
        x = [0x61707865, 0x3320646E, 0x79622D32, 0x6B206574] + key + [block & m32, block >> 32, 0, 0]
        y = list(x)
        for r in range(8):
            for c in range(4):
                at = [c, 4 + c, 8 + c, 12 + c] if r % 2 == 0 else [c, 4 + (c + 1) % 4, 8 + (c + 2) % 4, 12 + (c + 3) % 4]
                a, b, d, e = at
                for turn in (16, 12, 8, 7):
                    p, q, t = (a, b, e) if turn in (16, 8) else (d, e, b)
                    y[p] = (y[p] + y[q]) & m32
                    w = y[t] ^ y[p]
                    y[t] = ((w << turn) | (w >> (32 - turn))) & m32
        words += [(u + v) & m32 for u, v in zip(x, y)]
        block += 1
    return [((words[2 * k] | words[2 * k + 1] << 32) >> 11) * 2.0 ** -53 for k in range(count)]


def _exact_dynamic(case, seed):
    c = _dynamic(case, np.random.default_rng(seed))
    psi, bits = _zero_state(c.n), [0] * c.ncbits
    draws = iter(_draws(seed, 2 * c.ncbits))
    for kind, qs, vals, cnd in c.ops:
        if cnd is not None and bits[cnd[0]] != cnd[1]:
            continue
        if kind not in ("measure", "reset"):
            _apply(psi, kind, qs, vals)
            continue
        zero, one = _slices(psi, list(qs))
        p1 = float(one.abs().square().sum())
        if next(draws) < p1:
            one.div_(math.sqrt(p1))
            zero.zero_()
            if kind == "reset":
                zero.copy_(one)
                one.zero_()
            else:
                bits[vals[0]] = 1
        else:
            zero.div_(math.sqrt(max(1 - p1, 0)))
            one.zero_()
            if kind == "measure":
                bits[vals[0]] = 0
    return psi


def _exact_qft(case, seed):
    n, size = case["n"], 1 << case["n"]
    _, x = _qft(n, np.random.default_rng(seed))
    rev = int(format(x, "0%db" % n)[::-1], 2)
    psi = torch.empty(size, dtype=torch.complex128, device="cuda")
    step = 1 << 24
    for at in range(0, size, step):
        w = torch.arange(at, min(at + step, size), device="cuda")
        r = torch.zeros_like(w)
        for q in range(n):
            r |= ((w >> q) & 1) << (n - 1 - q)
        turn = ((r * rev) % size).double() * (2 * math.pi / size)
        psi[at:at + step] = torch.polar(torch.full_like(turn, 2.0 ** (-n / 2)), turn)
    return psi


def _signs(n, q):
    s = torch.ones(1 << n, dtype=torch.float64, device="cuda")
    s.view(-1, 2, 1 << q)[:, 1] = -1
    return s


def _exact_gradients(case, seed):
    """dE/dangle = Im <lambda|P|psi> after the gate exp(-i angle P / 2), gates undone in reverse."""
    n, layers = case["n"], case["layers"]
    theta = _theta(case, seed)
    a, b, _ = _observable(n, seed)
    sets = theta.shape[0]
    th = torch.tensor(theta, device="cuda").view(sets, layers, 3, n)

    def rotate(v, q, angle):  # ry by `angle` [sets]
        c, s = (f(angle / 2).view(-1, 1, 1) for f in (torch.cos, torch.sin))
        w = v.view(v.shape[0], -1, 2, 1 << q)
        x, y = w[:, :, 0].clone(), w[:, :, 1].clone()
        w[:, :, 0] = c * x - s * y
        w[:, :, 1] = s * x + c * y

    es, grads = [], []
    chunk = max(1, (1 << 25) >> n)
    signs = [_signs(n, q) for q in range(n)]
    for at in range(0, sets, chunk):
        t = th[at:at + chunk]
        psi = torch.zeros(t.shape[0], 1 << n, dtype=torch.complex128, device="cuda")
        psi[:, 0] = 1

        def phase(k):
            p = torch.zeros(t.shape[0], 1 << n, dtype=torch.float64, device="cuda")
            for q in range(n):
                p.addcmul_(t[:, k, 1, q, None], signs[q])
                p.addcmul_(t[:, k, 2, q, None], signs[q] * signs[(q + 1) % n])
            return torch.polar(torch.ones_like(p), p.mul_(-0.5))

        for k in range(layers):
            for q in range(n):
                rotate(psi, q, t[:, k, 0, q])
            psi *= phase(k)
        lam = torch.zeros_like(psi)
        for q in range(n):
            lam.addcmul_(psi, (a[q] * signs[q] * signs[(q + 1) % n]).to(psi.dtype))
            lam.view(lam.shape[0], -1, 2, 1 << q).add_(psi.view(lam.shape[0], -1, 2, 1 << q).flip(2), alpha=b[q])
        es.append((psi.conj() * lam).real.sum(1))
        g = torch.zeros_like(t)
        for k in reversed(range(layers)):
            z = (lam.conj() * psi).imag
            for q in range(n):
                g[:, k, 1, q] = z @ signs[q]
                g[:, k, 2, q] = z @ (signs[q] * signs[(q + 1) % n])
            p = phase(k).conj_physical_()
            psi *= p
            lam *= p
            del z, p
            for q in reversed(range(n)):
                u, v = (x.view(x.shape[0], -1, 2, 1 << q) for x in (psi, lam))
                # Y psi = (-i psi_1, i psi_0)
                g[:, k, 0, q] = ((v[:, :, 1].conj() * u[:, :, 0]).real - (v[:, :, 0].conj() * u[:, :, 1]).real).sum((1, 2))
                rotate(psi, q, -t[:, k, 0, q])
                rotate(lam, q, -t[:, k, 0, q])
        grads.append(g.reshape(t.shape[0], -1))
    return torch.cat(es), torch.cat(grads)


def _exact_mps(case, seed):
    c = _brickwork(case["n"], case["layers"], np.random.default_rng(seed))
    sites = [np.array([1, 0], dtype=complex).reshape(1, 2, 1) for _ in range(c.n)]
    for kind, qs, vals, _ in c.ops:
        m, q = _matrix(kind, vals), qs[0]
        if len(qs) == 1:
            sites[q] = np.einsum("st,ltr->lsr", m, sites[q])
            continue
        l, r = sites[q].shape[0], sites[q + 1].shape[2]
        both = np.einsum("lsm,mtr->lstr", sites[q], sites[q + 1])
        both = np.einsum("abst,lstr->labr", m.reshape(2, 2, 2, 2), both).reshape(2 * l, 2 * r)
        u, s, v = np.linalg.svd(both, full_matrices=False)
        keep = min(max(1, int(np.sum(s > 1e-12))), case["bond"])
        s2 = s[:keep] * (np.linalg.norm(s) / np.linalg.norm(s[:keep]))
        sites[q] = u[:, :keep].reshape(l, 2, keep)
        sites[q + 1] = (s2[:, None] * v[:keep]).reshape(keep, 2, r)
    w = torch.ones(1, 1, dtype=torch.complex128, device="cuda")  # qubit 0 is the lowest index bit
    for t in sites:
        t = torch.tensor(t, device="cuda")
        w = torch.einsum("il,lsr->sir", w, t).reshape(2 * w.shape[0], -1)
    return w.reshape(-1)


def exact(case, seed):
    f = case["family"]
    if f == "dynamic":
        return {"bits": None, "counts": None, "state": _exact_dynamic(case, seed)}
    if f == "brickwork":
        return {"counts": None, "state": _unitary(_brickwork(case["n"], case["layers"], np.random.default_rng(seed)))}
    if f == "qft":
        n = case["n"]
        return {"top": np.full(1 << min(10, n), 1.0 / (1 << min(10, n))), "state": _exact_qft(case, seed)}
    if f == "ragged":
        return [_unitary(c).cpu().numpy() for c in _ragged(case, np.random.default_rng(seed))]
    if f in ("gradient", "gradients"):
        e, g = _exact_gradients(case, seed)
        return {"energy": float(e[0]), "gradient": g[0].cpu().numpy()} if f == "gradient" else {"energy": e, "gradient": g}
    if f == "mps":
        return {"state": _exact_mps(case, seed)}
    return None
