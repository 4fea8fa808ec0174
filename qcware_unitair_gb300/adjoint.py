"""Adjoint differentiation of expectation values of parameterised circuits.

    pc = ParamCircuit(n, num_params)
    pc.ry(q, p); pc.rz(q, p); pc.cz(a, b); pc.end_layer()
    H = PauliSum(n).z(0).xx(0, 1, coeff=0.5)
    values = expectation(pc, params, H)            # (B,) float64, autograd
    values.mean().backward()                       # adjoint sweep, no tape

Rotations follow unitair's convention (src/unitair/gates/gates.py:6-91):
RX(theta) = exp_x(theta / 2) = exp(-i theta/2 X), likewise RY, RZ; the angle
of a rotation is ``scale * params[b, p]`` per batch entry b.

The forward pass runs the circuit as a fused program (one HBM pass per
stage) and keeps the state at checkpoints every ~sqrt(depth) layers.  The
backward pass starts from lambda = H psi_L (gbsv_pauli_sum_apply_host) and
walks the gates in reverse, in stages as the forward pass has them
(gbsv_adjoint_stage_regs, or gbsv_adjoint_stage where a stage has no register
plan): for each rotation the gradient Im<l|P|psi>, summed in FP64 beyond a
thread, then U^dag on psi and lambda.  A rotation or gate outside the stages
is a launch of its own on both states.  At each checkpoint the uncomputed psi
is replaced by the stored forward state, so rounding drift never accumulates
over more than one segment.
This replaces torch autograd through unitair's apply_operator, which keeps
every intermediate state (one per gate) alive for the backward pass.
"""
from __future__ import annotations

import math
from typing import Dict, List, Optional, Sequence

import numpy as np
import torch

import ctypes

from . import _core, _lib, states

ctypes_int32 = ctypes.c_int32
from .circuits import gate_matrix
from .fusion import CTRL, DENSE, DIAG, Circuit

GEN = {"X": 0, "Y": 1, "Z": 2}


class PauliSum:
    """H = sum_k c_k P_k with real c_k and Pauli strings P_k."""

    def __init__(self, num_qubits: int):
        self.num_qubits = num_qubits
        self.terms: List[tuple] = []  # (coeff, {qubit: 'X'|'Y'|'Z'})

    def add(self, coeff: float, paulis: Dict[int, str]) -> "PauliSum":
        for q, p in paulis.items():
            if p not in "XYZ" or not 0 <= q < self.num_qubits:
                raise ValueError(f"bad Pauli {p} on qubit {q}")
        self.terms.append((float(coeff), dict(paulis)))
        return self

    def z(self, q, coeff=1.0):
        return self.add(coeff, {q: "Z"})

    def xx(self, a, b, coeff=1.0):
        return self.add(coeff, {a: "X", b: "X"})

    def term_array(self) -> np.ndarray:
        """Records matching gbsv_pauli_term_t (xmask, zmask, re, im)."""
        n = self.num_qubits
        dt = np.dtype([("x", "<u8"), ("z", "<u8"), ("re", "<f8"),
                       ("im", "<f8")])
        out = np.zeros(len(self.terms), dtype=dt)
        xs, zs, res, ims = [], [], [], []
        for c, ps in self.terms:
            xm = zm = ny = 0
            for q, p in ps.items():
                bit = 1 << (n - 1 - q)
                if p in "XY":
                    xm |= bit
                if p in "ZY":
                    zm |= bit
                ny += p == "Y"
            # c * i^ny
            xs.append(xm)
            zs.append(zm)
            res.append((c, 0.0, -c, 0.0)[ny & 3])
            ims.append((0.0, c, 0.0, -c)[ny & 3])
        out["x"], out["z"], out["re"], out["im"] = xs, zs, res, ims
        return out

    def dense(self) -> np.ndarray:
        """2^n x 2^n matrix (small n; for tests)."""
        n = self.num_qubits
        P = {"I": np.eye(2), "X": np.array([[0, 1], [1, 0]]),
             "Y": np.array([[0, -1j], [1j, 0]]), "Z": np.diag([1, -1])}
        H = np.zeros((2 ** n, 2 ** n), dtype=np.complex128)
        for c, ps in self.terms:
            m = np.array([[1.0]])
            for q in range(n):
                m = np.kron(m, P[ps.get(q, "I")])
            H += c * m
        return H


def hardware_efficient_ansatz(num_qubits: int, layers: int):
    """Each layer applies U = RY(theta) RZ(phi) to every qubit (RZ acts
    first), then a ring of CZ(q, q+1 mod n).  Parameter (layer, qubit, k)
    has index (layer * n + qubit) * 2 + k, k = 0 for theta and 1 for phi,
    i.e. a (B, layers, n, 2) tensor reshaped to (B, layers * n * 2)."""
    n = num_qubits
    pc = ParamCircuit(n, layers * n * 2)
    for l in range(layers):
        for q in range(n):
            base = (l * n + q) * 2
            pc.rz(q, base + 1)
            pc.ry(q, base + 0)
        for q in range(n):
            if n > 1 and (q + 1 < n or n > 2):
                pc.cz(q, (q + 1) % n)
        pc.end_layer()
    return pc


class ParamCircuit:
    """Rotations driven by a (B, num_params) parameter tensor plus fixed
    gates; ``end_layer`` marks layer boundaries for checkpointing."""

    def __init__(self, num_qubits: int, num_params: int):
        self.num_qubits = num_qubits
        self.num_params = num_params
        self.ops: list = []
        self.layer_ends: List[int] = []

    def _rot(self, gen, q, p, scale):
        if not 0 <= p < self.num_params:
            raise ValueError(f"parameter index {p} out of range")
        if not 0 <= q < self.num_qubits:
            raise ValueError(f"qubit {q} out of range")
        self.ops.append(("rot", gen, int(q), int(p), float(scale)))
        return self

    def rx(self, q, p, scale=1.0): return self._rot("X", q, p, scale)
    def ry(self, q, p, scale=1.0): return self._rot("Y", q, p, scale)
    def rz(self, q, p, scale=1.0): return self._rot("Z", q, p, scale)

    def gate(self, matrix, qubits, kind: Optional[str] = None):
        m = torch.as_tensor(np.asarray(matrix, dtype=np.complex128))
        self.ops.append(("fixed", m, tuple(int(q) for q in qubits), kind))
        return self

    def h(self, q): return self.gate(gate_matrix("H"), [q], DENSE)
    def cz(self, a, b): return self.gate(gate_matrix("CZ"), [a, b], DIAG)
    def cnot(self, c, t): return self.gate(gate_matrix("CNOT"), [c, t], CTRL)

    def end_layer(self):
        self.layer_ends.append(len(self.ops))
        return self

    # -- segments for checkpoints ---------------------------------------
    def segments(self, every: Optional[int] = None) -> List[tuple]:
        """Op ranges [a, b) between checkpoints, every ~sqrt(depth)
        layers (or ~sqrt(ops) without layer marks)."""
        ends = [e for e in self.layer_ends if 0 < e <= len(self.ops)]
        if ends and ends[-1] != len(self.ops):
            ends.append(len(self.ops))
        if not ends:
            k = every or max(1, int(math.ceil(math.sqrt(len(self.ops)))))
            ends = list(range(k, len(self.ops), k)) + [len(self.ops)]
        else:
            k = every or max(1, int(math.ceil(math.sqrt(len(ends)))))
            ends = ends[k - 1::k] if len(ends) > k else []
            if not ends or ends[-1] != len(self.ops):
                ends.append(len(self.ops))
        out, a = [], 0
        for e in ends:
            if e > a:
                out.append((a, e))
            a = e
        return out or [(0, 0)]

    # -- building blocks ---------------------------------------------------
    def _segment_circuit(self, a, b, params, dtype) -> Circuit:
        """Ops [a, b) as a Circuit with per-state rotation matrices."""
        c = Circuit(self.num_qubits)
        B = params.shape[0]
        for op in self.ops[a:b]:
            if op[0] == "fixed":
                _, m, qs, kind = op
                c.append(m, qs, kind)
                continue
            _, gen, q, p, scale = op
            th = params[:, p].detach().to(torch.float64) * (0.5 * scale)
            cs, sn = torch.cos(th), torch.sin(th)
            z = torch.zeros_like(cs)
            if gen == "X":
                m = torch.stack([torch.complex(cs, z), torch.complex(z, -sn),
                                 torch.complex(z, -sn), torch.complex(cs, z)],
                                -1)
                kind = DENSE
            elif gen == "Y":
                m = torch.stack([torch.complex(cs, z), torch.complex(-sn, z),
                                 torch.complex(sn, z), torch.complex(cs, z)],
                                -1)
                kind = DENSE
            else:
                m = torch.stack([torch.complex(cs, -sn), torch.complex(z, z),
                                 torch.complex(z, z), torch.complex(cs, sn)],
                                -1)
                kind = DIAG
            c.append(m.reshape(B, 2, 2).to(dtype), [q], kind)
        return c


# placeholder rotation matrices fix each rotation's record kind when a
# forward program is planned once per circuit structure: a generic complex
# 2x2 for X (dense), a real one for Y (real 2x2), a diagonal for Z
_PLACEHOLDER = {
    "X": torch.tensor([[0.6 + 0.2j, 0.1 - 0.3j], [0.4 + 0.1j, 0.7 - 0.2j]],
                      dtype=torch.complex128),
    "Y": torch.tensor([[0.8, -0.6], [0.6, 0.8]], dtype=torch.complex128),
    "Z": torch.tensor([[0.6 - 0.8j, 0], [0, 0.6 + 0.8j]],
                      dtype=torch.complex128),
}


def _forward_program(pc: ParamCircuit, a: int, b: int, B: int, dtype, dev,
                     fuse: bool):
    """(Program, its rotations, their gates) for ops [a, b) with B states,
    planned once per structure.  Each call only fills a pool of gate values
    (_call_pool)."""
    key = (a, b, B, dtype, str(dev), fuse)
    cache = pc.__dict__.setdefault("_fwd_cache", {})
    if key in cache:
        return cache[key]
    c = Circuit(pc.num_qubits)
    rots = []
    for op in pc.ops[a:b]:
        if op[0] == "fixed":
            _, m, qs, kind = op
            c.append(m, qs, kind)
            continue
        _, gen, q, p, scale = op
        ph = _PLACEHOLDER[gen].expand(B, 2, 2).clone()
        c.append(ph, [q], DIAG if gen == "Z" else DENSE)
        rots.append((c.gates[-1], op))
    prog = c.compile(dtype, dev, fuse=fuse, native=False)
    idx, which = [], []
    for g, op in rots:
        if fuse:
            off, nv = prog.gate_pool[id(g)]
        else:
            off, nv = None, 4
        which.append((op[1], op[3], op[4], off, nv))
    if fuse and which:
        _rotation_records(prog, which, B)
    cache[key] = (prog, which, rots)
    return cache[key]


def _rotation_values(which, params, B, dtype):
    """All rotations' pool entries, flattened in ``which`` order (rotation,
    state, entry), from torch operations: what _write_rotations is tested
    against."""
    dev = params.device
    gen = torch.tensor(["XYZ".index(w[0]) for w in which], device=dev)
    pidx = torch.tensor([w[1] for w in which], device=dev)
    half = torch.tensor([0.5 * w[2] for w in which], dtype=torch.float64,
                        device=dev)
    nv = torch.tensor([w[4] for w in which], device=dev)
    keep = (torch.arange(4, device=dev)[None, None, :] <
            nv[:, None, None]).expand(len(which), B, 4)
    th = params[:, pidx].to(torch.float64) * half          # (B, R)
    c, s = torch.cos(th).T, torch.sin(th).T                 # (R, B)
    z = torch.zeros_like(c)
    isx, isy = (gen == 0)[:, None], (gen == 1)[:, None]
    isz4 = ((gen == 2) & (nv == 4))[:, None]
    # entry k of each rotation, real and imaginary parts (R, B)
    re0, im0 = c, torch.where(isx | isy, z, -s)
    re1 = torch.where(isy, -s, torch.where(isx | isz4, z, c))
    im1 = torch.where(isx, -s, torch.where(isy | isz4, z, s))
    re2, im2 = torch.where(isy, s, z), torch.where(isx, -s, z)
    re3, im3 = c, torch.where(isz4, s, z)
    re = torch.stack([re0, re1, re2, re3], -1)
    im = torch.stack([im0, im1, im2, im3], -1)
    return torch.complex(re, im).to(dtype)[keep]


ROT_DTYPE = np.dtype([("gen", "<i4"), ("nv", "<i4"), ("pidx", "<i4"),
                      ("pad", "<i4"), ("off", "<i8"), ("half", "<f8")])


def _circuit_params(pc, params: torch.Tensor) -> torch.Tensor:
    """The circuit's parameters, (B, num_params): the kernels index a row by
    that number, and read past one that is shorter."""
    if params.dim() != 2 or params.shape[1] < pc.num_params:
        raise ValueError(f"params must be (B, {pc.num_params}), got "
                         f"{tuple(params.shape)}")
    return params[:, :pc.num_params]


def _real_params(params: torch.Tensor) -> torch.Tensor:
    """Parameters as the kernels read them: contiguous float32/float64."""
    p = _core.dense(params.detach())
    if p.dtype not in (torch.float32, torch.float64):
        p = p.to(torch.float64)
    return p


def _rotation_records(prog, which, B):
    """The records that fill a pool for this program, on the device: its
    rotations, then copies of what lies between them, four entries a
    thread."""
    from .fusion import _to_device
    recs = [(GEN[gen], nv, pi, 0, off, 0.5 * scale)
            for gen, pi, scale, off, nv in which]
    at = 0
    for off, end in sorted((off, off + B * nv) for *_, off, nv in which) + [
            (prog.pool.numel(), 0)]:
        while at < off:
            n = min(off - at, 4 * B)
            recs.append((3, n, 0, 0, at, 0.0))
            at += n
        at = max(at, end)
    prog._rot_recs = _to_device(np.array(recs, ROT_DTYPE).view(np.uint8),
                                prog.pool.device)
    prog._rot_count = len(recs)
    prog._rot_uploads = _core.Uploads([prog._rot_recs], prog.pool.device)


def _write_rotations(prog, which, p, pool=None):
    """Every rotation's matrices written by one kernel (sin and cos in FP64):
    into the program's own pool, or all of ``pool``."""
    dev, stream = p.device, _core.stream_of(p.device)
    prog._rot_uploads.use(dev, stream)
    prog._uploads.use(dev, stream)
    own = pool is None
    rc = _lib.load().gbsv_rotation_pool(
        p.data_ptr(), _core.real_code(p.dtype), p.shape[1], p.shape[0],
        prog._rot_recs.data_ptr(), len(which) if own else prog._rot_count,
        None if own else prog.pool.data_ptr(),
        (prog.pool if own else pool).data_ptr(),
        _core.complex_code(prog.dtype), stream)
    _lib.check(rc, "rotation_values")


def _call_pool(prog, which, p):
    """The gate values of one evaluation.  The program is shared by every
    evaluation of its circuit, on whatever stream or thread, so what depends
    on the parameters is not kept in it."""
    if not which:
        return prog.pool
    pool = torch.empty_like(prog.pool)
    _write_rotations(prog, which, p, pool)
    return pool


def _initial_state(n, B, dtype, device, psi0):
    if psi0 is None:
        s = torch.zeros(B, 2 ** n, dtype=dtype, device=device)
        s[:, 0] = 1
        return s
    s = psi0.to(device=device, dtype=dtype)
    if s.dim() == 1:
        s = s.expand(B, -1)
    return _core.dense(s.reshape(B, 2 ** n))


def _forward(pc: ParamCircuit, params, dtype, psi0, checkpoints: bool,
             fuse: bool = True):
    """Run the circuit; return (psi_L, [psi at each segment start]), each in
    memory of its own but the first, which may be psi0 (a checkpoint that no
    sweep goes back to, or the result where there is nothing to run)."""
    n, B = pc.num_qubits, params.shape[0]
    dev = params.device
    psi = _initial_state(n, B, dtype, dev, psi0)
    saved = []
    p = _real_params(params)
    # whether psi's memory is this function's and not the caller's psi0
    own = psi0 is None or psi.data_ptr() != psi0.data_ptr()
    for a, b in pc.segments():
        # a segment leaves its checkpoint where it is and writes elsewhere
        keep = checkpoints and fuse and b > a
        if checkpoints:
            saved.append(psi if keep else psi.clone())
        if b <= a:
            continue
        inplace = own and not keep
        own = True
        if not fuse:
            prog = pc._segment_circuit(a, b, params, dtype).compile(
                dtype, dev, fuse=False)
            psi = prog.run(psi, inplace=inplace)
            continue
        prog, which, _ = _forward_program(pc, a, b, B, dtype, dev, fuse)
        psi = prog._run(psi, inplace, None, _call_pool(prog, which, p))
    return psi, saved


def _pauli_apply(H: PauliSum, psi: torch.Tensor, out: torch.Tensor):
    terms = H.term_array()
    n = H.num_qubits
    rc = _lib.load().gbsv_pauli_sum_apply_host(
        psi.data_ptr(), out.data_ptr(), _core.complex_code(psi.dtype), n,
        psi.numel() >> n, terms.ctypes.data, len(terms),
        _core.stream_of(psi.device))
    _lib.check(rc, "pauli_sum_apply")
    return out


def pauli_expectation(H: PauliSum, psi: torch.Tensor) -> torch.Tensor:
    """<psi|H|psi> per state (float64, FP64 accumulation)."""
    psi = _core.dense(psi)
    lam = torch.empty_like(psi)
    _pauli_apply(H, psi, lam)
    return _real_inner(psi, lam)


def _real_inner(a, b):
    """Re <a|b> per row with the FP64 accumulator returned unrounded."""
    ip = states._inner_product_kernel(a, b, out_dtype=torch.complex128)
    return ip.real


def _backward_sweep(pc, params, H, psi_L, saved, dtype):
    n, B = pc.num_qubits, params.shape[0]
    dev = params.device
    N = 2 ** n
    buf = torch.empty(2, B, N, dtype=dtype, device=dev)
    psi, lam = buf[0], buf[1]
    psi.copy_(psi_L)
    _pauli_apply(H, psi, lam)
    grads = torch.zeros(B, pc.num_params, dtype=torch.float64, device=dev)
    p = _real_params(params)
    L = _lib.load()
    code = _core.complex_code(dtype)
    acode = _core.real_code(p.dtype)
    esz = p.element_size()
    stream = _core.stream_of(dev)
    nbytes = int(L.gbsv_adjoint_scratch_bytes(B, n))
    scratch = torch.empty(max(nbytes, 16), dtype=torch.uint8, device=dev)
    both = buf.view(2 * B, N)
    # every fixed gate's adjoint, moved to the device in one transfer
    fixed = [op for op in pc.ops if op[0] == "fixed"]
    dag = {}
    if fixed:
        flat = [_core.dense(op[1].conj().T).reshape(-1) for op in fixed]
        host = torch.cat(flat).to(dtype)
        if dev.type == "cuda":
            host = host.pin_memory()
        devbuf = host.to(dev, non_blocking=True)
        off = 0
        for op, f in zip(fixed, flat):
            d = op[1].shape[-1]
            dag[id(op)] = devbuf[off:off + f.numel()].view(d, d)
            off += f.numel()
    segs = pc.segments() if saved else [(0, len(pc.ops))]
    for si in range(len(segs) - 1, -1, -1):
        a, b = segs[si]
        for op in reversed(pc.ops[a:b]):
            if op[0] == "rot":
                _, gen, q, pi, scale = op
                rc = L.gbsv_adjoint_rotation_step(
                    psi.data_ptr(), lam.data_ptr(), code, n, B, q, GEN[gen],
                    p.data_ptr() + pi * esz, acode, pc.num_params, scale,
                    grads.data_ptr() + pi * 8, pc.num_params, scale,
                    scratch.data_ptr(), nbytes, stream)
                _lib.check(rc, "adjoint_rotation_step")
            else:
                _, m, qs, _kind = op
                md = dag[id(op)]
                wide = not _core.inplace_ok(dtype, len(qs), n)
                dst = torch.empty_like(both) if wide else both
                rc = L.gbsv_apply_operator(
                    both.data_ptr(), dst.data_ptr(), code, n, 2 * B, N,
                    md.data_ptr(), 0, _lib.qubit_array(qs), len(qs), stream)
                _lib.check(rc, "apply_operator")
                if wide:
                    both.copy_(dst)
        if saved:
            psi.copy_(saved[si])  # re-anchor at the forward checkpoint
    return grads


def evaluate(pc: ParamCircuit, params: torch.Tensor, H: PauliSum,
             psi0: Optional[torch.Tensor] = None,
             dtype=torch.complex64) -> torch.Tensor:
    """Forward only: <psi|H|psi> per batch entry (float64), no gradient."""
    _core.require_cuda(params)
    params = _circuit_params(pc, params)
    psi_L, _ = _forward(pc, params, dtype, psi0, False)
    return pauli_expectation(H, psi_L)


ADJOP_DTYPE = np.dtype([("kind", "<i4"), ("gen", "<i4"), ("bit", "<i4"),
                        ("slot", "<i4"), ("pidx", "<i4"), ("pad", "<i4"),
                        ("scale", "<f8")])


def _adjop_dtype():
    from .fusion import FG_DTYPE
    return np.dtype(ADJOP_DTYPE.descr + [("g", FG_DTYPE)])


def _plan_backward(pc: ParamCircuit, a: int, b: int, dtype, dev, m: int,
                   device_ops: bool = True):
    """Fused backward stages for ops [a, b) walked in reverse: a list of
    ("stage", launch args) / ("rot", op) / ("fixed", op) entries.  Depends
    only on the circuit's structure, so it is cached per circuit."""
    from .fusion import CircuitGate, FG_DTYPE, _record, _to_device, plan
    n = pc.num_qubits
    ops = list(reversed(pc.ops[a:b]))
    stand = []
    dummy = torch.zeros(2, 2, dtype=torch.complex128)
    for op in ops:
        if op[0] == "rot":
            stand.append(CircuitGate(dummy, (op[2],),
                                     DIAG if op[1] == "Z" else DENSE))
        else:
            _, mat, qs, kind = op
            stand.append(CircuitGate(mat.conj().transpose(-1, -2), qs,
                                     kind or DENSE))
    index = {id(g): op for g, op in zip(stand, ops)}
    c_min = min(4 if dtype == torch.complex64 else 3, m)
    out = []
    AD = _adjop_dtype()
    for kind, item in plan(stand, n, m, c_min):
        if kind == "plain":
            op = index[id(item)]
            out.append(("rot" if op[0] == "rot" else "fixed", op))
            continue
        tile = item.tile
        c = 0
        while c in tile:
            c += 1
        c = min(c, m)
        order = list(range(c)) + sorted(p for p in tile if p >= c)
        local = {p: i for i, p in enumerate(order)}
        G = len(item.gates)
        recs = np.zeros(G, dtype=AD)  # filled by column: no per-record
        kinds = np.zeros(G, np.int32)  # structured-array promotion
        gens = np.zeros(G, np.int32)
        bits = np.zeros(G, np.int32)
        slots = np.zeros(G, np.int32)
        pidxs = np.zeros(G, np.int32)
        scales = np.zeros(G, np.float64)
        pool, slot_p, slot_s = [], [], []
        pool_len = 0
        for i, g in enumerate(item.gates):
            op = index[id(g)]
            if op[0] == "rot":
                _, gen, q, pi, scale = op
                pos = n - 1 - q
                gens[i] = GEN[gen]
                bits[i] = local[pos] if pos in local else -1 - pos
                slots[i], pidxs[i], scales[i] = len(slot_p), pi, scale
                slot_p.append(pi)
                slot_s.append(scale)
            else:
                rec, vals = _record(g, n, local, None)
                v = vals.reshape(-1).to(dtype)
                rec["mat"], rec["mat_bstride"] = pool_len, 0
                pool.append(v)
                pool_len += v.numel()
                kinds[i] = 1
                recs["g"][i] = rec
        recs["kind"], recs["gen"], recs["bit"] = kinds, gens, bits
        recs["slot"], recs["pidx"], recs["scale"] = slots, pidxs, scales
        args = {
            "c": c, "positions": (ctypes_int32 * m)(*order),
            "records": recs, "host_pool": None,
            "params": (slot_p, slot_s), "num_ops": G,
            "pool": (torch.cat(pool) if pool else torch.zeros(1, dtype=dtype)
                     ).to(dev),
            "num_slots": len(slot_p)}
        if device_ops:
            _device_stage(args, dev)
        out.append(("stage", args))
    return out


def _device_stage(args, dev):
    """What gbsv_adjoint_stage reads from the device."""
    from .fusion import _to_device
    slot_p, slot_s = args["params"]
    args["ops"] = _to_device(args["records"].view(np.uint8), dev)
    args["slot_param"] = torch.tensor(list(slot_p) or [0], dtype=torch.int32,
                                      device=dev)
    args["slot_scale"] = torch.tensor(list(slot_s) or [0.0],
                                      dtype=torch.float64, device=dev)


def _plan_backward_native(pc: ParamCircuit, a: int, b: int, dtype, dev,
                          m: int, device_ops: bool = True):
    """_plan_backward with the stages planned by gbsv_plan (C++) and the
    adjoint records assembled by column: the same stages, records and
    values (one pool for all stages instead of one per stage)."""
    from .fusion import DESC_DTYPE, _KIND_CODE, native_plan
    n = pc.num_qubits
    ops = list(reversed(pc.ops[a:b]))
    G = len(ops)
    desc = np.zeros(max(1, G), dtype=DESC_DTYPE)
    parts = [np.eye(2, dtype=np.complex128).reshape(-1)]  # rotations' stand-in
    off = 4
    kinds, nqs, q0s, q1s, offs = [], [], [], [], []
    is_rot = np.zeros(G, dtype=bool)
    gens = np.zeros(G, np.int32)
    pidxs = np.zeros(G, np.int32)
    scales = np.zeros(G, np.float64)
    dag = {}  # adjoints of repeated fixed matrices (the same object)
    for i, op in enumerate(ops):
        if op[0] == "rot":
            _, gen, q, pi, scale = op
            kinds.append(_KIND_CODE[DIAG if gen == "Z" else DENSE])
            nqs.append(1)
            q0s.append(q)
            q1s.append(0)
            offs.append(0)
            is_rot[i] = True
            gens[i], pidxs[i], scales[i] = GEN[gen], pi, scale
        else:
            _, mat, qs, kind = op
            md = dag.get(id(mat))
            if md is None:
                md = np.ascontiguousarray(
                    np.conj(mat.detach().cpu().numpy()).T,
                    dtype=np.complex128).reshape(-1)
                dag[id(mat)] = md
            kinds.append(_KIND_CODE[kind or DENSE])
            nqs.append(len(qs))
            q0s.append(qs[0])
            q1s.append(qs[1] if len(qs) > 1 else 0)
            offs.append(off)
            parts.append(md)
            off += md.size
    if G:
        desc["kind"][:G], desc["nq"][:G] = kinds, nqs
        desc["q0"][:G], desc["q1"][:G], desc["mat"][:G] = q0s, q1s, offs
        desc["num_batch"][:G] = 1
    mats = np.ascontiguousarray(np.concatenate(parts))
    c_min = min(4 if dtype == torch.complex64 else 3, m)
    nat = native_plan(None, n, m, c_min, 0, True, dtype, desc[:G], mats)
    recs = nat["records"]
    pool = torch.from_numpy(nat["pool"]).to(dev) if len(nat["pool"]) else \
        torch.zeros(1, dtype=dtype, device=dev)
    AD = _adjop_dtype()
    out = []
    nxt = 0  # next gate index not yet placed
    for op in nat["ops"]:
        t, first, count = int(op["type"]), int(op["first"]), int(op["count"])
        if t == 0:
            assert first == nxt
            src = ops[first]
            out.append(("rot" if src[0] == "rot" else "fixed", src))
            nxt = first + 1
            continue
        idx = np.arange(nxt, nxt + count)
        nxt += count
        r = recs[first:first + count]
        rot = is_rot[idx]
        ad = np.zeros(count, dtype=AD)
        ad["kind"] = np.where(rot, 0, 1)
        ad["gen"] = gens[idx]
        ad["bit"] = np.where(rot, r["b0"], 0)
        ad["slot"] = np.where(rot, np.cumsum(rot) - 1, 0)
        ad["pidx"] = np.where(rot, pidxs[idx], 0)
        ad["scale"] = np.where(rot, scales[idx], 0.0)
        ad["g"][~rot] = r[~rot]
        args = {
            "c": int(op["contiguous"]),
            "positions": (ctypes_int32 * m)(
                *[int(x) for x in op["positions"][:m]]),
            "records": ad, "host_pool": nat["pool"],
            "params": (pidxs[idx][rot], scales[idx][rot]),
            "num_ops": count,
            "pool": pool,
            "num_slots": int(rot.sum())}
        if device_ops:
            _device_stage(args, dev)
        out.append(("stage", args))
    assert nxt == G
    return out


REGOP_DTYPE = np.dtype([("type", "<i4"), ("slot", "<i4"), ("nq", "<i4"),
                        ("signs", "<i4"), ("k", "<i4", 2), ("t", "<u4", 2),
                        ("o", "<i4", 2), ("mat", "<i8"), ("cmask", "<u8"),
                        ("cval", "<u8")])
LAYOUT_DTYPE = np.dtype([("rb", "i1", 4), ("tb", "i1", 12), ("first", "<i4"),
                         ("count", "<i4"), ("pad", "<i4", 2)])
ANGLE_DTYPE = np.dtype([("pidx", "<i4"), ("pad", "<i4"), ("half", "<f8")])


def _register_plan(entries, m: int, dtype, dev):
    """The register form of a segment's stages: per stage its ops and layouts
    (byte offsets into one device buffer), the segment's rotations in slot
    order and the chains that join the slots of one parameter.  None where
    the stages do not fit it (small tiles, per-state gates)."""
    from .fusion import _to_device
    L = _lib.load()
    code = _core.complex_code(dtype)
    rb = int(L.gbsv_adjoint_register_bits(code))
    if not rb + 5 <= m <= rb + 8:
        return None
    pieces, size = [], 0

    def add(arr):
        nonlocal size
        raw = np.ascontiguousarray(arr).view(np.uint8).reshape(-1)
        pad = -len(raw) % 64
        at = size
        pieces.append(raw)
        if pad:
            pieces.append(np.zeros(pad, np.uint8))
        size += len(raw) + pad
        return at

    stages, params, scales = [], [], []
    for kind, st in entries:
        if kind != "stage":
            continue
        G = st["num_ops"]
        rec = np.ascontiguousarray(st["records"])
        ops = np.empty(max(4 * G, 1), REGOP_DTYPE)
        lays = np.zeros(max(G, 1), LAYOUT_DTYPE)
        hp = st["host_pool"]
        nops, count = ctypes.c_int(0), ctypes.c_int(0)
        rc = L.gbsv_adjoint_layouts(
            rec.ctypes.data, G, m, rb,
            hp.ctypes.data if hp is not None and len(hp) else None, code,
            ops.ctypes.data, ctypes.byref(nops), lays.ctypes.data, len(lays),
            ctypes.byref(count))
        if rc == _lib.GBSV_ERR_UNSUPPORTED:
            return None
        _lib.check(rc, "adjoint_layouts")
        stages.append((add(ops[:max(nops.value, 1)]), nops.value,
                       add(lays[:max(count.value, 1)]), count.value,
                       len(params)))
        params.extend(int(x) for x in st["params"][0])
        scales.extend(float(x) for x in st["params"][1])
    total = len(params)
    rots = np.zeros(max(total, 1), ANGLE_DTYPE)
    prev = np.full(max(total, 1), -1, np.int32)
    nxt = np.full(max(total, 1), -1, np.int32)
    last = {}
    for k, p in enumerate(params):
        rots[k] = (p, 0, 0.5 * scales[k])
        if p in last:
            prev[k] = last[p]
            nxt[last[p]] = k
        last[p] = k
    at = {"rots": add(rots), "prev": add(prev), "next": add(nxt),
          "param": add(np.array(params or [0], np.int32)),
          "scale": add(np.array(scales or [0.0], np.float64))}
    most = max([st["num_slots"] for kind, st in entries if kind == "stage"],
               default=0)
    return {"buf": _to_device(np.concatenate(pieces), dev),
            "stages": stages, "at": at, "total": total, "most": most}


# gradient partials kept before they are summed (bytes)
_PARTIAL_BYTES = 64 << 20


def _segment_plan(pc, a, b, dtype, dev, m):
    """Entries of the backward sweep over ops [a, b), their register plan
    (None: not all of them have one) and what of them is on the device, made
    once per circuit."""
    cache = pc.__dict__.setdefault("_adj_cache", {})
    key = (a, b, dtype, str(dev), m)
    if key not in cache:
        host = all(op[0] == "rot" or not op[1].is_cuda for op in pc.ops[a:b])
        plan = (_plan_backward_native if host else _plan_backward)(
            pc, a, b, dtype, dev, m, device_ops=False)
        regs = _register_plan(plan, m, dtype, dev)
        stages = [st for kind, st in plan if kind == "stage"]
        if regs is None:
            for st in stages:
                _device_stage(st, dev)
        held = {id(t): t for st in stages for t in st.values()
                if isinstance(t, torch.Tensor)}
        uploads = _core.Uploads([*held.values()] + (
            [regs["buf"]] if regs is not None else []), dev)
        cache[key] = (plan, regs, uploads)
    return cache[key]


def _backward_fused(pc, params, H, psi_L, saved, dtype, lam=None):
    """The adjoint sweep with fused backward stages (see the kernel
    gbsv_adjoint_stage): one read and write of psi and lambda per stage.
    With ``lam`` (H psi_L from the forward pass) the sweep runs in lam,
    psi_L and the checkpoints themselves; without, it leaves them alone."""
    n, B = pc.num_qubits, params.shape[0]
    dev = params.device
    N = 2 ** n
    m = min(12 if dtype == torch.complex64 else 11, n)
    segs = pc.segments() if saved else [(0, len(pc.ops))]
    plans = [_segment_plan(pc, a, b, dtype, dev, m) for a, b in segs]
    # gates outside the stages run on psi and lambda as one batch
    owned = lam is not None and all(
        entry[0] in ("stage", "rot") for plan, *_ in plans for entry in plan)
    if owned:
        psi = psi_L
    else:
        buf = torch.empty(2, B, N, dtype=dtype, device=dev)
        both = buf.view(2 * B, N)
        psi = buf[0].copy_(psi_L)
        lam = (_pauli_apply(H, psi, buf[1]) if lam is None
               else buf[1].copy_(lam))
    grads = torch.zeros(B, pc.num_params, dtype=torch.float64, device=dev)
    p = _real_params(params)
    L = _lib.load()
    code = _core.complex_code(dtype)
    pcode = _core.real_code(p.dtype)
    stream = _core.stream_of(dev)
    tiles = B << (n - m)
    scratch = partial = None
    for si in range(len(segs) - 1, -1, -1):
        entries, regs, uploads = plans[si]
        uploads.use(dev, stream)
        if regs is not None and regs["total"]:
            buf0, at = regs["buf"].data_ptr(), regs["at"]
            total = regs["total"]
            angles = torch.empty(B, total, 2, dtype=torch.float64, device=dev)
            rc = L.gbsv_adjoint_angles(
                p.data_ptr(), pcode, pc.num_params, B, buf0 + at["rots"],
                total, angles.data_ptr(), stream)
            _lib.check(rc, "adjoint_angles")
            room = min(total, max(regs["most"],
                                  _PARTIAL_BYTES // (8 * tiles)))
            if partial is None or partial.numel() < room * tiles:
                partial = torch.empty(room * tiles, dtype=torch.float64,
                                      device=dev)
        first = slot = 0  # slots [first, slot) are in partial, unsummed

        def sum_slots():
            rc = L.gbsv_adjoint_grad_sum(
                partial.data_ptr(), first, slot, B, 1 << (n - m),
                buf0 + at["param"], buf0 + at["scale"], buf0 + at["prev"],
                buf0 + at["next"], grads.data_ptr(), pc.num_params, stream)
            _lib.check(rc, "adjoint_grad_sum")

        index = 0
        for entry in entries:
            if entry[0] == "stage" and regs is not None:
                st = entry[1]
                op_at, G, lay_at, nlay, slot = regs["stages"][index]
                index += 1
                ns = st["num_slots"]
                if ns and slot + ns - first > room:
                    sum_slots()
                    first = slot
                base = regs["buf"].data_ptr()
                rc = L.gbsv_adjoint_stage_regs(
                    psi.data_ptr(), lam.data_ptr(), code, n, B, m, st["c"],
                    st["positions"], base + op_at, G, base + lay_at, nlay,
                    st["pool"].data_ptr(),
                    angles.data_ptr() if ns else None, regs["total"], slot,
                    ns, partial.data_ptr() + (slot - first) * tiles * 8
                    if ns else None, stream)
                _lib.check(rc, "adjoint_stage")
                slot += ns
            elif entry[0] == "stage":
                st = entry[1]
                need = st["num_slots"] * (tiles + 2 * B) * 8
                if need and (scratch is None or scratch.numel() < need):
                    scratch = torch.empty(need, dtype=torch.uint8, device=dev)
                rc = L.gbsv_adjoint_stage(
                    psi.data_ptr(), lam.data_ptr(), code, n, B, m, st["c"],
                    st["positions"], st["ops"].data_ptr(), st["num_ops"],
                    st["pool"].data_ptr(), p.data_ptr(), pcode,
                    pc.num_params, st["num_slots"],
                    st["slot_param"].data_ptr(), st["slot_scale"].data_ptr(),
                    grads.data_ptr(),
                    scratch.data_ptr() if need else None, need, stream)
                _lib.check(rc, "adjoint_stage")
            elif entry[0] == "rot":
                _, gen, q, pi, scale = entry[1]
                nbytes = int(L.gbsv_adjoint_scratch_bytes(B, n))
                sc = torch.empty(max(nbytes, 16), dtype=torch.uint8,
                                 device=dev)
                rc = L.gbsv_adjoint_rotation_step(
                    psi.data_ptr(), lam.data_ptr(), code, n, B, q, GEN[gen],
                    p.data_ptr() + pi * p.element_size(), pcode,
                    pc.num_params, scale, grads.data_ptr() + pi * 8,
                    pc.num_params, scale, sc.data_ptr(), nbytes, stream)
                _lib.check(rc, "adjoint_rotation_step")
            else:
                _, m_, qs, _k = entry[1]
                md = _core.dense(m_.conj().T).to(device=dev, dtype=dtype)
                wide = not _core.inplace_ok(dtype, len(qs), n)
                dst = torch.empty_like(both) if wide else both
                rc = L.gbsv_apply_operator(
                    both.data_ptr(), dst.data_ptr(), code, n, 2 * B, N,
                    md.data_ptr(), 0, _lib.qubit_array(qs), len(qs), stream)
                _lib.check(rc, "apply_operator")
                if wide:
                    both.copy_(dst)
        if slot > first:
            sum_slots()
        if saved and si > 0:  # re-anchor at the forward checkpoint
            psi = saved[si] if owned else psi.copy_(saved[si])
    return grads


def expectation_and_grad(pc: ParamCircuit, params: torch.Tensor,
                         H: PauliSum, psi0: Optional[torch.Tensor] = None,
                         dtype=torch.complex64, checkpoints: bool = True,
                         fuse: bool = True):
    """(values (B,), grads (B, num_params)), both float64.  ``fuse=False``
    runs the forward pass one kernel per gate.  Parameters beyond the
    circuit's are not looked at."""
    _core.require_cuda(params)
    params = _circuit_params(pc, params)
    psi_L, saved = _forward(pc, params, dtype, psi0, checkpoints, fuse)
    lam = _pauli_apply(H, psi_L, torch.empty_like(psi_L))
    values = _real_inner(psi_L, lam)
    if fuse:
        grads = _backward_fused(pc, params, H, psi_L, saved, dtype, lam)
    else:
        grads = _backward_sweep(pc, params, H, psi_L, saved, dtype)
    return values, grads


class _Expectation(torch.autograd.Function):
    @staticmethod
    def forward(ctx, params, pc, H, psi0, dtype, checkpoints):
        psi_L, saved = _forward(pc, params, dtype, psi0, checkpoints)
        lam = _pauli_apply(H, psi_L, torch.empty_like(psi_L))
        ctx.pc, ctx.H, ctx.dtype = pc, H, dtype
        ctx.psi_L, ctx.saved = psi_L, saved
        # H psi_L, which starts the backward sweep.  That pass then allocates
        # no state: one more is held between the passes, two fewer during the
        # second, and on 32 states of 16 qubits five copies (24 us) and an
        # application of H (30 us) are saved.
        ctx.lam = lam if ctx.needs_input_grad[0] else None
        ctx.save_for_backward(params)
        return _real_inner(psi_L, lam)

    @staticmethod
    def backward(ctx, g):
        (params,) = ctx.saved_tensors
        grads = _backward_fused(ctx.pc, params, ctx.H, ctx.psi_L,
                                ctx.saved, ctx.dtype, ctx.lam)
        ctx.psi_L = ctx.saved = ctx.lam = None
        out = (g.to(torch.float64).unsqueeze(-1) * grads).to(params.dtype)
        return out, None, None, None, None, None


def expectation(pc: ParamCircuit, params: torch.Tensor, H: PauliSum,
                psi0: Optional[torch.Tensor] = None, dtype=torch.complex64,
                checkpoints: bool = True) -> torch.Tensor:
    """<psi(params)|H|psi(params)> per batch entry (float64), differentiable
    with respect to ``params`` by the adjoint method."""
    _core.require_cuda(params)
    if params.dim() != 2 or params.shape[1] != pc.num_params:
        raise ValueError(f"params must be (B, {pc.num_params}), got "
                         f"{tuple(params.shape)}")
    return _Expectation.apply(params, pc, H, psi0, dtype, checkpoints)
