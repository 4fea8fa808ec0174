"""The fused all-qubit kernel (csrc/allq.cu) against the oracle at the edges
of its tiles: the smallest states, several states in a tile, one to three
passes, a last CTA that is partly empty, broadcast states, per-state and
per-qubit operators, views at an odd offset.

Tolerance: an amplitude goes through n complex 2x2 products of unitary
matrices; each rounds by at most about 4 * 2^-24 of the pair's norm, so n
products of random signs stay below 8 * sqrt(n) * 2^-24 of the state's
largest amplitudes (norm 1, at most about 1)."""
import numpy as np
import pytest
import torch

import qcware_unitair_gb300 as ug
from oracle import oracle

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _unitaries(rng, shape):
    a = rng.normal(size=shape + (2, 2)) + 1j * rng.normal(size=shape + (2, 2))
    return np.linalg.qr(a)[0].astype(np.complex64)


def _states(rng, shape, n):
    a = rng.normal(size=shape + (2 ** n,)) + 1j * rng.normal(
        size=shape + (2 ** n,))
    a /= np.linalg.norm(a, axis=-1, keepdims=True)
    return a.astype(np.complex64)


def _reference(ops, psi, n, each):
    out = psi.astype(np.complex128)
    for q in range(n):
        m = ops[..., q, :, :] if each else ops
        out = oracle.apply_operator(m.astype(np.complex128), [q], out)
    return out


def _tol(n):
    return 8 * np.sqrt(n) * 2.0 ** -24


# 4-8 qubits: many states per tile (and a last tile partly empty); 9-12: one
# layout overlaps the previous; 13 and 16: a high pass of 1 and 4 bits; 17:
# 5 (both layouts); 20: 8; 21: three passes
@pytest.mark.parametrize("n,batch", [
    (4, 1), (4, 257), (5, 131), (6, 65), (7, 33), (8, 1), (8, 17), (9, 9),
    (10, 5), (11, 3), (12, 3), (13, 2), (16, 3), (17, 2), (20, 1), (21, 1)])
@pytest.mark.parametrize("each", [False, True])
@pytest.mark.parametrize("per_state", [False, True])
def test_all_qubits_matches_oracle(n, batch, each, per_state):
    rng = np.random.default_rng(1000 * n + batch)
    b = (batch,)
    ops = _unitaries(rng, (b if per_state else ()) + ((n,) if each else ()))
    psi = _states(rng, b, n)
    fn = ug.apply_each_qubit if each else ug.apply_all_qubits
    got = fn(torch.from_numpy(ops).to(DEV), torch.from_numpy(psi).to(DEV))
    ref = _reference(ops, psi, n, each)
    assert got.shape == ref.shape
    assert np.abs(got.cpu().numpy() - ref).max() <= _tol(n)


# structured operators (real, RX-like, diagonal) take shorter forms: equal to
# the gate-by-gate kernel bit for bit, also where an amplitude is not finite
@pytest.mark.parametrize("n", [6, 12, 18])
@pytest.mark.parametrize("gate", ["H", "RX", "RZ", "full"])
def test_structured_operators_equal_the_gate_loop(n, gate):
    rng = np.random.default_rng(n)
    t = torch.tensor(0.7)
    m = {"H": ug.gates.hadamard(), "RX": ug.gates.rx(t),
         "RZ": ug.gates.rz(t),
         "full": torch.from_numpy(_unitaries(rng, ()))}[gate].to(DEV)
    psi = torch.from_numpy(_states(rng, (2,), n)).to(DEV)
    psi[1, 5] = complex(float("inf"), 0.0)
    psi[1, 9] = complex(0.0, float("nan"))
    loop = psi
    for q in range(n):
        loop = ug.apply_operator(m, [q], loop)
    got = ug.apply_all_qubits(m, psi)
    assert torch.equal(torch.isfinite(got), torch.isfinite(loop))
    assert torch.equal(got[0], loop[0])
    a, b = torch.view_as_real(got[1]), torch.view_as_real(loop[1])
    assert torch.equal(torch.nan_to_num(a, 7.0), torch.nan_to_num(b, 7.0))


@pytest.mark.parametrize("n", [5, 10, 14])
def test_all_qubits_broadcast_state_and_odd_offset(n):
    rng = np.random.default_rng(n)
    ops = _unitaries(rng, (6,))
    psi = _states(rng, (), n)
    buf = torch.zeros(2 ** n + 1, dtype=torch.complex64, device=DEV)
    buf[1:] = torch.from_numpy(psi)
    got = ug.apply_all_qubits(torch.from_numpy(ops).to(DEV), buf[1:])
    ref = _reference(ops, psi, n, False)
    assert np.abs(got.cpu().numpy() - ref).max() <= _tol(n)


# Gradients against complex128 autograd through the per-qubit loop.  Per
# amplitude the FP32 states differ from complex128 by about 4 sqrt(2 n)
# 2^-24 of the state's norm (forward and adjoint), sums are exact beside
# that, and a sum over B states and n qubits grows like the reference's.
@pytest.mark.parametrize("n,batch", [(9, 9), (10, 4), (11, 3), (12, 2),
                                     (13, 2), (17, 2), (20, 1), (22, 1)])
@pytest.mark.parametrize("each", [False, True])
@pytest.mark.parametrize("form", ["shared", "per_state", "broadcast_state",
                                  "operator_only"])
def test_all_qubits_gradients(n, batch, each, form):
    rng = np.random.default_rng(n)
    b = (batch,)
    ops = torch.from_numpy(_unitaries(
        rng, (b if form in ("per_state", "broadcast_state") else ()) +
        ((n,) if each else ()))).to(DEV)
    psi = torch.from_numpy(_states(
        rng, () if form == "broadcast_state" else b, n)).to(DEV)
    w = torch.from_numpy(_states(rng, b, n)).to(DEV)

    def loss(m, s, wide):
        if wide:
            out = s
            for q in range(n):
                out = ug.apply_operator(m[..., q, :, :] if each else m, [q],
                                        out)
        else:
            out = (ug.apply_each_qubit if each else ug.apply_all_qubits)(m, s)
        return (w.to(out.dtype).conj() * out).sum(-1).abs().square().sum()

    grads = []
    for dt in (torch.complex64, torch.complex128):
        m = ops.to(dt, copy=True).requires_grad_()
        s = psi.to(dt, copy=True).requires_grad_(form != "operator_only")
        loss(m, s, dt == torch.complex128).backward()
        grads.append((m.grad, s.grad))
    tol = 16 * np.sqrt(2 * n) * 2.0 ** -24
    for got, ref in zip(*grads):
        if ref is None:
            assert got is None
            continue
        assert got.shape == ref.shape and got.dtype == torch.complex64
        off = torch.linalg.vector_norm(got.to(ref.dtype) - ref)
        assert off <= tol * torch.linalg.vector_norm(ref) * n


def test_all_qubits_gradient_state_only_and_unused():
    n, rng = 14, np.random.default_rng(3)
    m = torch.from_numpy(_unitaries(rng, (2,))).to(DEV)
    s = torch.from_numpy(_states(rng, (2,), n)).to(DEV).requires_grad_()
    w = torch.from_numpy(_states(rng, (2,), n)).to(DEV)
    out = ug.apply_all_qubits(m, s)
    out.backward(w)
    ref = ug.apply_all_qubits(m.conj().transpose(-1, -2), w)
    assert torch.equal(s.grad, ref)
