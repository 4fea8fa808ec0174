"""Timed workloads of the engine, through its public functions.

Every case is one of the kinds below at some size; ``listed()`` gives one or
two of each, ``draw()`` others of the same ranges.

  gates        a run of gates applied one at a time (apply_operator), the
               loop that circuit code on this API is made of: from batches of
               small states, where a call's latency counts, to one state of
               several GiB, where memory bandwidth does
  rotations    a layer of per-state RX, RY and RZ on every qubit and a CNOT
               ladder on a batch of states, each state with its own angles
  trotter      time evolution of a batch under a diagonal energy and a
               transverse field: apply_phase, apply_all_qubits and the energy
  qaoa_grad    a variational optimiser's step: forward and backward of a
               QAOA energy with respect to every angle (autograd)
  gate_grad    a training step of general k-qubit unitaries against target
               states: forward and backward with respect to the operators and
               the input states (autograd)
  fused        a circuit compiled once and run as fused stages (Program.run)
  adjoint      expectation and gradient of a hardware-efficient ansatz by the
               adjoint method
  operator     a 3-qubit gate and a general 4- to 6-qubit block on random
               qubits
  observables  what is read out of a batch of states: probabilities, norms,
               overlaps, a diagonal observable
  shots        a CZ layer, a qubit exchange and cyclic shift, a Toffoli, and
               basis states sampled from the result
"""
import math

import numpy as np
import torch

import qcware_unitair_gb300 as ug
from qcware_unitair_gb300 import adjoint as ad
from qcware_unitair_gb300 import measurement

DEV = "cuda"


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # 64 small states: the smallest calls, bound by launches and host work
        _case("gates", n=12, batch=64, gates=8, name="gates_12q_x64"),
        # one large state: bound by memory bandwidth
        _case("gates", n=28, batch=1, gates=6, name="gates_28q"),
        # double precision, as numerical checks and long circuits ask for it
        _case("gates", n=24, batch=3, gates=8, dtype="complex128",
              name="gates_24q_x3_c128"),
        # a batch of parameter settings evaluated at once
        _case("rotations", n=16, batch=256, name="rotations_16q_x256"),
        # an evolution step of a few mid-sized states
        _case("trotter", n=20, batch=7, steps=2, name="trotter_20q_x7"),
        # an optimiser's step over several starting points
        _case("qaoa_grad", n=14, batch=16, layers=3, name="qaoa_grad_14q_x16"),
        # training general two-qubit gates on a few states
        _case("gate_grad", n=18, batch=5, k=2, gates=6, per_state=False,
              name="gate_grad_18q_x5"),
        # a mid-sized random circuit in fused stages
        _case("fused", n=26, batch=1, gates=120, name="fused_26q"),
        # a variational batch with gradients
        _case("adjoint", n=16, batch=32, layers=4, name="adjoint_16q_x32"),
        # Toffoli-sized gates and a wider block
        _case("operator", n=25, batch=2, k=5, name="operator_25q_k5"),
        # reading out a batch of states
        _case("observables", n=20, batch=33, name="observables_20q_x33"),
        # entangling layer and sampling of one state
        _case("shots", n=24, batch=1, samples=100000, name="shots_24q"),
    ]


def _case(kind, n, batch, dtype="complex64", name=None, **more):
    c = {"kind": kind, "n": n, "batch": batch, "dtype": dtype, **more}
    if name is not None:
        c["name"] = name
    return c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gates", "gates", "rotations", "trotter", "qaoa_grad",
                       "gate_grad", "fused", "adjoint", "operator",
                       "observables", "shots"])
    # one case in four in double precision (sampling and the fused circuit of
    # tensor-core stages are used in single precision)
    dtype = "complex128" if rng.random() < 0.25 else "complex64"

    def size(n_lo, n_hi, log_most, log_least=0):
        """Qubits over their range, then a batch (odd ones too) so that the
        whole is at most 2^log_most amplitudes (half of that in double
        precision) and at least 2^log_least."""
        most = log_most - (1 if dtype == "complex128" else 0)
        n = rng.randint(n_lo, min(n_hi, most))
        lo = 2 ** max(0, min(log_least, most) - n)
        return n, max(1, _log_int(rng, lo, 2 ** (most - n)))

    if kind == "gates":
        n, b = size(8, 28, 27, 12)
        return _case(kind, n, b, dtype, gates=rng.randint(4, 10))
    if kind == "rotations":
        n, b = size(8, 20, 24, 14)
        return _case(kind, n, b, dtype)
    if kind == "trotter":
        n, b = size(10, 24, 24, 14)
        return _case(kind, n, b, dtype, steps=rng.randint(1, 4))
    if kind == "qaoa_grad":
        n, b = size(8, 18, 19, 11)
        return _case(kind, n, b, dtype, layers=rng.randint(1, 4))
    if kind == "gate_grad":
        n, b = size(8, 22, 21, 11)
        return _case(kind, n, b, dtype, k=rng.choice([1, 2, 2, 3]),
                     gates=rng.randint(3, 8), per_state=rng.random() < 0.3)
    if kind == "fused":
        n, b = size(10, 26, 26, 16)
        return _case(kind, n, b, dtype, gates=_log_int(rng, 40, 160))
    if kind == "adjoint":
        n, b = size(8, 18, 21, 13)
        return _case(kind, n, b, dtype, layers=rng.randint(2, 6))
    if kind == "operator":
        # double precision runs on the FP64 units: smaller states
        n, b = size(10, 26, 26 if dtype == "complex64" else 23, 14)
        return _case(kind, n, b, dtype, k=rng.choice([4, 5, 6]))
    if kind == "observables":
        n, b = size(10, 26, 26, 14)
        return _case(kind, n, b, dtype)
    n = rng.randint(12, 26)
    return _case(kind, n, 1, "complex64", samples=_log_int(rng, 1000, 1000000))


# ----------------------------------------------------------------- inputs --
def _dtype(case):
    return getattr(torch, case["dtype"])


def _real(case):
    return torch.float64 if case["dtype"] == "complex128" else torch.float32


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _states(g, batch, n, dtype):
    """Random normalised states, (batch, 2^n), or (2^n,) for a single one."""
    s = torch.randn((batch, 2 ** n), generator=g, dtype=dtype, device=DEV)
    s /= torch.linalg.vector_norm(s, dim=-1, keepdim=True)
    return s if batch > 1 else s[0]


def _rotation(axis, theta, dtype):
    """exp(-i theta/2 P) for angles of any shape -> (*shape, 2, 2)."""
    t = torch.as_tensor(theta, dtype=torch.float64) / 2
    c, s = torch.cos(t).to(torch.complex128), torch.sin(t).to(torch.complex128)
    z = torch.zeros_like(c)
    rows = {"X": [c, -1j * s, -1j * s, c], "Y": [c, -s, s, c],
            "Z": [c - 1j * s, z, z, c + 1j * s]}[axis]
    return torch.stack(rows, -1).reshape(t.shape + (2, 2)).to(dtype)


def _named_gates():
    h = 2 ** -0.5
    f = {"H": [[h, h], [h, -h]], "X": [[0, 1], [1, 0]],
         "Y": [[0, -1j], [1j, 0]], "Z": [[1, 0], [0, -1]],
         "S": [[1, 0], [0, 1j]],
         "T": [[1, 0], [0, complex(h, h)]],
         "CNOT": [[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 0, 1], [0, 0, 1, 0]],
         "CZ": [[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 1, 0], [0, 0, 0, -1]],
         "SWAP": [[1, 0, 0, 0], [0, 0, 1, 0], [0, 1, 0, 0], [0, 0, 0, 1]]}
    return {k: torch.tensor(v, dtype=torch.complex128) for k, v in f.items()}


def _circuit(n, count, seed):
    """Uniform gates of {H, X, Y, Z, S, T, RX, RY, RZ, CNOT, CZ, SWAP} on
    uniform distinct qubits: (name, host complex128 matrix, qubits)."""
    rng = np.random.default_rng(seed)
    fixed = _named_gates()
    names = list(fixed) + ["RX", "RY", "RZ"]
    out = []
    for _ in range(count):
        name = names[int(rng.integers(len(names)))]
        k = 2 if name in ("CNOT", "CZ", "SWAP") else 1
        qs = tuple(int(q) for q in rng.choice(n, size=k, replace=False))
        m = fixed[name] if name in fixed else _rotation(
            name[1], float(rng.uniform(0, 2 * math.pi)), torch.complex128)
        out.append((name, m, qs))
    return out


def _unitaries(g, shape, k, dtype):
    """Random unitaries (QR of complex normals), shape + (2^k, 2^k)."""
    d = 2 ** k
    a = torch.randn(tuple(shape) + (d, d), generator=g,
                    dtype=torch.complex128, device=DEV)
    return torch.linalg.qr(a)[0].to(dtype).contiguous()


def _cut_values(n, seed, real):
    """MaxCut value of every bit string for a random graph of about 3n/2
    edges, as a (2^n,) real tensor."""
    rng = np.random.default_rng(seed)
    idx = torch.arange(2 ** n, device=DEV)
    out = torch.zeros(2 ** n, dtype=real, device=DEV)
    for a in range(n):
        for b in {(a + 1) % n, int(rng.integers(n))} - {a}:
            out += ((idx >> (n - 1 - a)) ^ (idx >> (n - 1 - b))) & 1
    return out


def _zz_energy(n, seed, real):
    """sum_i J_i Z_i Z_i+1 + h_i Z_i of every bit string, J and h normal."""
    rng = np.random.default_rng(seed)
    idx = torch.arange(2 ** n, device=DEV)
    z = [1 - 2 * ((idx >> (n - 1 - q)) & 1).to(real) for q in range(n)]
    out = torch.zeros(2 ** n, dtype=real, device=DEV)
    for q in range(n):
        out += float(rng.normal()) * z[q]
        if q + 1 < n:
            out += float(rng.normal()) * z[q] * z[q + 1]
    return out


def _inputs(case, seed):
    """The case's tensors, from the seed alone."""
    kind, n, b = case["kind"], case["n"], case["batch"]
    dt, real, g = _dtype(case), _real(case), _generator(seed)
    rng = np.random.default_rng(seed)
    x = {}
    if kind in ("gates", "fused"):
        x["psi"] = _states(g, b, n, dt)
        x["gates"] = [(name, m.to(dt) if kind == "gates" else m, qs)
                      for name, m, qs in _circuit(n, case["gates"], seed)]
        if kind == "gates":
            x["gates"] = [(a, m.to(DEV), q) for a, m, q in x["gates"]]
    elif kind == "rotations":
        x["psi"] = _states(g, b, n, dt)
        shape = (b, n) if b > 1 else (n,)
        for axis in "XYZ":
            th = torch.rand(shape, generator=g, dtype=real, device=DEV)
            x[axis] = _rotation(axis, th * (2 * math.pi), dt)
        x["cnot"] = _named_gates()["CNOT"].to(device=DEV, dtype=dt)
    elif kind == "trotter":
        x["psi"] = _states(g, b, n, dt)
        x["energy"] = _zz_energy(n, seed, real)
        step = 0.05 + 0.1 * float(rng.random())
        x["angles"] = step * x["energy"]
        x["field"] = _rotation("X", torch.tensor(2 * step), dt).to(DEV)
    elif kind == "qaoa_grad":
        x["cut"] = _cut_values(n, seed, real)
        for name in ("gamma", "beta"):
            x[name] = torch.rand((b, case["layers"]), generator=g, dtype=real,
                                 device=DEV)
    elif kind == "gate_grad":
        x["psi"] = _states(g, b, n, dt)
        x["target"] = _states(g, b, n, dt)
        x["qubits"] = [tuple(int(q) for q in rng.choice(
            n, size=case["k"], replace=False)) for _ in range(case["gates"])]
        shape = (b,) if case["per_state"] and b > 1 else ()
        x["ops"] = [_unitaries(g, shape, case["k"], dt) for _ in x["qubits"]]
    elif kind == "adjoint":
        x["params"] = torch.randn((b, case["layers"] * n * 2), generator=g,
                                  dtype=real, device=DEV)
    elif kind == "operator":
        x["psi"] = _states(g, b, n, dt)
        x["ops"] = [(_unitaries(g, (), k, dt),
                     tuple(int(q) for q in rng.choice(n, size=k,
                                                      replace=False)))
                    for k in (3, case["k"])]
    elif kind == "observables":
        x["psi"], x["other"] = _states(g, b, n, dt), _states(g, b, n, dt)
        x["diagonal"] = _zz_energy(n, seed, real)
    else:
        x["psi"] = _states(g, b, n, dt)
        qs = [int(q) for q in rng.permutation(n)]
        x["pairs"] = torch.tensor([[i, (i + 1) % n] for i in range(0, n, 2)],
                                  device=DEV)
        x["pair_list"] = x["pairs"].tolist()
        x["swap"], x["shift"] = (qs[0], qs[1]), 1 + int(rng.integers(n - 1))
        x["toffoli"] = ([qs[2], qs[3]], qs[4])
        x["seed"] = int(rng.integers(1 << 30))
    return x


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    x = _inputs(case, seed)
    x["case"] = dict(case)
    if kind == "fused":
        # the program that a caller compiles once for its circuit
        c = ug.Circuit(n)
        for name, m, qs in x["gates"]:
            c.append(m, list(qs), {"Z": "diag", "S": "diag", "T": "diag",
                                   "RZ": "diag", "CZ": "diag",
                                   "CNOT": "ctrl"}.get(name, "dense"))
        x["program"] = c.compile(_dtype(case), torch.device(DEV, 0))
    elif kind == "qaoa_grad":
        x["hadamard"] = ug.gates.hadamard(device=DEV, dtype=_dtype(case))
    elif kind == "adjoint":
        x["circuit"] = ad.hardware_efficient_ansatz(n, case["layers"])
        h = ad.PauliSum(n)
        for q in range(n):
            h.z(q)
        for q in range(n - 1):
            h.xx(q, q + 1, 0.5)
        x["observable"] = h
    return x


# -------------------------------------------------------------------- run --
def run(x):
    case = x["case"]
    return _RUN[case["kind"]](x, case)


def _run_gates(x, case):
    psi = x["psi"]
    for _, m, qs in x["gates"]:
        psi = ug.apply_operator(m, qs, psi)
    return psi


def _run_rotations(x, case):
    psi = x["psi"]
    for axis in "XYZ":
        psi = ug.apply_each_qubit(x[axis], psi)
    for q in range(case["n"] - 1):
        psi = ug.apply_operator(x["cnot"], [q, q + 1], psi)
    return psi


def _run_trotter(x, case):
    psi = x["psi"]
    for _ in range(case["steps"]):
        psi = ug.apply_phase(x["angles"], psi)
        psi = ug.apply_all_qubits(x["field"], psi)
    return psi, ug.diag_expectation_value(x["energy"], psi)


def _run_qaoa_grad(x, case):
    n, dt = case["n"], _dtype(case)
    gamma = x["gamma"].detach().requires_grad_()
    beta = x["beta"].detach().requires_grad_()
    psi = ug.unit_vector(0, n, device=torch.device(DEV, 0), dtype=dt)
    psi = ug.apply_all_qubits(x["hadamard"], psi)
    psi = psi.expand(case["batch"], 2 ** n)
    for l in range(case["layers"]):
        psi = ug.apply_phase(gamma[:, l, None] * x["cut"], psi)
        psi = ug.apply_all_qubits(ug.gates.exp_x(beta[:, l], dtype=dt), psi)
    energy = ug.diag_expectation_value(x["cut"], psi)
    energy.sum().backward()
    return energy.detach(), psi.detach(), gamma.grad, beta.grad


def _run_gate_grad(x, case):
    psi0 = x["psi"].detach().requires_grad_()
    ops = [m.detach().requires_grad_() for m in x["ops"]]
    psi = psi0
    for m, qs in zip(ops, x["qubits"]):
        psi = ug.apply_operator(m, qs, psi)
    # the operators need not stay unitary while they are trained
    fidelity = (ug.inner_product(x["target"], psi).abs().square() /
                ug.norm_squared(psi))
    (1 - fidelity).sum().backward()
    return fidelity.detach(), psi0.grad, [m.grad for m in ops]


def _run_fused(x, case):
    return x["program"].run(x["psi"])


def _run_adjoint(x, case):
    p = x["params"].detach().requires_grad_()
    values = ad.expectation(x["circuit"], p, x["observable"],
                            dtype=_dtype(case))
    values.mean().backward()
    return values.detach(), p.grad


def _run_operator(x, case):
    psi = x["psi"]
    for m, qs in x["ops"]:
        psi = ug.apply_operator(m, qs, psi)
    return psi


def _run_observables(x, case):
    psi = x["psi"]
    return {"p": ug.abs_squared(psi), "norm": ug.norm_squared(psi),
            "overlap": ug.inner_product(x["other"], psi),
            "mean": ug.diag_expectation_value(x["diagonal"], psi)}


def _run_shots(x, case):
    psi = ug.multi_cz(x["pairs"], x["psi"])
    psi = ug.swap(psi, x["swap"])
    psi = ug.roll_qubits(psi, x["shift"])
    psi = ug.multi_controlled_x(psi, *x["toffoli"])
    return psi, measurement.sample(psi, case["samples"], seed=x["seed"])


_RUN = {"gates": _run_gates, "rotations": _run_rotations,
        "trotter": _run_trotter, "qaoa_grad": _run_qaoa_grad,
        "gate_grad": _run_gate_grad, "fused": _run_fused,
        "adjoint": _run_adjoint, "operator": _run_operator,
        "observables": _run_observables, "shots": _run_shots}


# ------------------------------------------------------------------- work --
def work(case):
    """Bytes: what each public call reads and writes, once; a fused circuit
    and an adjoint sweep are one call.  Flops: of the dense gates."""
    kind, n, b = case["kind"], case["n"], case["batch"]
    amps = b * 2 ** n
    amp = 16 if case["dtype"] == "complex128" else 8
    state, real = amps * amp, amp // 2
    if kind == "gates":
        return {"bytes": 2 * state * case["gates"],
                "flops": 14 * amps * case["gates"]}
    if kind == "rotations":
        return {"bytes": 2 * state * (3 + n - 1),
                "flops": 14 * amps * 3 * n}
    if kind == "trotter":
        return {"bytes": (4 * state + 2 ** n * real) * case["steps"] + state,
                "flops": (14 * n + 10) * amps * case["steps"]}
    if kind == "qaoa_grad":
        # forward: phase and mixer; backward: the same and their saved
        # states; angles written, read and their gradients
        layer = 4 * state + 6 * state + 4 * amps * real
        return {"bytes": layer * case["layers"] + 3 * state,
                "flops": 3 * (14 * n + 10) * amps * case["layers"]}
    if kind == "gate_grad":
        return {"bytes": state * (2 + 3) * case["gates"] + 6 * state,
                "flops": 3 * 8 * 2 ** case["k"] * amps * case["gates"]}
    if kind == "fused":
        return {"bytes": 2 * state, "flops": 14 * amps * case["gates"]}
    if kind == "adjoint":
        return {"bytes": 6 * state,
                "flops": 14 * amps * case["layers"] * 2 * n * 4}
    if kind == "operator":
        return {"bytes": 4 * state, "flops": 8 * amps * (8 + 2 ** case["k"])}
    if kind == "observables":
        return {"bytes": 5 * state + amps * real + 2 ** n * real,
                "flops": 20 * amps}
    return {"bytes": 9 * state + 8 * case["samples"], "flops": 4 * amps}


# ------------------------------------------------------------------ exact --
def _apply(m, qubits, psi, n):
    """A gate on (*batch, 2^n) states: the target axes moved to the front of
    each state, one matrix product, and back."""
    k = len(qubits)
    batch = psi.shape[:-1]
    order = sorted(range(k), key=lambda j: qubits[j])
    dims, prev = [], 0
    for j in order:
        dims += [2 ** (qubits[j] - prev), 2]
        prev = qubits[j] + 1
    dims.append(2 ** (n - prev))
    nb = len(batch)
    place = {j: nb + 2 * i + 1 for i, j in enumerate(order)}
    front = [place[j] for j in range(k)]
    rest = [nb + 2 * i for i in range(k + 1)]
    perm = list(range(nb)) + front + rest
    t = psi.reshape(tuple(batch) + tuple(dims)).permute(perm)
    shape = t.shape
    out = torch.matmul(m, t.reshape(tuple(batch) + (2 ** k, -1)))
    back = [perm.index(i) for i in range(len(perm))]
    return out.reshape(shape).permute(back).reshape(psi.shape)


def _up(t):
    return t.to(torch.complex128 if t.is_complex() else torch.float64)


def exact(case, seed):
    """What run() returns, in complex128 torch on the same inputs."""
    kind, n, b = case["kind"], case["n"], case["batch"]
    x = _inputs(case, seed)
    if kind in ("gates", "fused", "operator"):
        psi = _up(x["psi"])
        todo = [(m, qs) for _, m, qs in x["gates"]] if "gates" in x \
            else x["ops"]
        for m, qs in todo:
            psi = _apply(_up(m).to(DEV), qs, psi, n)
        return psi
    if kind == "rotations":
        psi = _up(x["psi"])
        for axis in "XYZ":
            ops = _up(x[axis])
            for q in range(n):
                psi = _apply(ops[..., q, :, :], (q,), psi, n)
        for q in range(n - 1):
            psi = _apply(_up(x["cnot"]), (q, q + 1), psi, n)
        return psi
    if kind == "trotter":
        psi = _up(x["psi"])
        phase = torch.exp(-1j * _up(x["angles"]))
        for _ in range(case["steps"]):
            psi = phase * psi
            for q in range(n):
                psi = _apply(_up(x["field"]), (q,), psi, n)
        return psi, (_up(x["energy"]) * psi.abs().square()).sum(-1)
    if kind == "qaoa_grad":
        gamma = _up(x["gamma"]).requires_grad_()
        beta = _up(x["beta"]).requires_grad_()
        cut = _up(x["cut"])
        psi = torch.full((b, 2 ** n), 2 ** (-n / 2), dtype=torch.complex128,
                         device=DEV)
        for l in range(case["layers"]):
            psi = torch.exp(-1j * gamma[:, l, None] * cut) * psi
            c, s = torch.cos(beta[:, l]) + 0j, torch.sin(beta[:, l]) * 1j
            m = torch.stack([c, -s, -s, c], -1).reshape(b, 2, 2)
            for q in range(n):
                psi = _apply(m, (q,), psi, n)
        energy = (cut * psi.abs().square()).sum(-1)
        energy.sum().backward()
        return energy.detach(), psi.detach(), gamma.grad, beta.grad
    if kind == "gate_grad":
        psi0 = _up(x["psi"]).requires_grad_()
        ops = [_up(m).requires_grad_() for m in x["ops"]]
        psi = psi0
        for m, qs in zip(ops, x["qubits"]):
            psi = _apply(m, qs, psi, n)
        fidelity = ((_up(x["target"]).conj() * psi).sum(-1).abs().square() /
                    psi.abs().square().sum(-1))
        (1 - fidelity).sum().backward()
        return fidelity.detach(), psi0.grad, [m.grad for m in ops]
    if kind == "adjoint":
        p = _up(x["params"]).requires_grad_()
        th = p.reshape(b, case["layers"], n, 2)
        idx = torch.arange(2 ** n, device=DEV)
        z = [1.0 - 2.0 * ((idx >> (n - 1 - q)) & 1) for q in range(n)]
        ring = torch.ones(2 ** n, dtype=torch.float64, device=DEV)
        for q in range(n):
            r = (q + 1) % n
            ring *= 1 - (1 - z[q]) * (1 - z[r]) / 2
        psi = torch.zeros((b, 2 ** n), dtype=torch.complex128, device=DEV)
        psi[:, 0] = 1
        for l in range(case["layers"]):
            for q in range(n):
                y, f = th[:, l, q, 0] / 2, th[:, l, q, 1] / 2
                e = torch.exp(-1j * f)
                c, s = torch.cos(y), torch.sin(y)
                m = torch.stack([c * e, -s / e, s * e, c / e], -1)
                psi = _apply(m.reshape(b, 2, 2), (q,), psi, n)
            psi = psi * ring
        values = (sum(z) * psi.abs().square()).sum(-1)
        for q in range(n - 1):
            t = psi.reshape(b, 2 ** q, 4, -1)
            values = values + 0.5 * (t.conj() * t.flip(2)).sum((1, 2, 3)).real
        values.mean().backward()
        return values.detach(), p.grad
    psi = _up(x["psi"])
    if kind == "observables":
        p = psi.abs().square()
        return {"p": p, "norm": p.sum(-1),
                "overlap": (_up(x["other"]).conj() * psi).sum(-1),
                "mean": (_up(x["diagonal"]) * p).sum(-1)}
    gate = {k: _up(v).to(DEV) for k, v in _named_gates().items()}
    for pair in x["pair_list"]:
        psi = _apply(gate["CZ"], tuple(pair), psi, n)
    psi = _apply(gate["SWAP"], x["swap"], psi, n)
    # out[a_0 .. a_n-1] = in[a_k .. a_k-1]: the last n - k index bits come
    # first in the input
    psi = psi.reshape(2 ** (n - x["shift"]), 2 ** x["shift"]).T.reshape(-1)
    toffoli = torch.eye(8, dtype=torch.complex128, device=DEV)
    toffoli[6:, 6:] = gate["X"]
    psi = _apply(toffoli, tuple(x["toffoli"][0]) + (x["toffoli"][1],), psi, n)
    return psi, None
