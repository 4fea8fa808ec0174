"""Lazily conjugated (and negated) tensors: conj() and the gradients autograd
hands to a backward set a bit on the tensor and leave its memory alone.  Every
entry point gives what it gives for the resolved values, on the native route
and on the Python one (numpy integers as qubits, operator batches that
broadcast onto another state batch).  Exact: the same kernels on the same
values; gradients as close as the order of their sums allows (1e-5, 1e-12)."""
import numpy as np
import pytest
import torch

import qcware_unitair_gb300 as ug
from qcware_unitair_gb300 import adjoint, measurement, simulation, states
from qcware_unitair_gb300.fusion import Circuit

pytestmark = pytest.mark.gpu
C64, C128 = torch.complex64, torch.complex128
DEV = "cuda"


def rand(*shape, dtype=C64, seed=0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return torch.randn(*shape, dtype=dtype, generator=g).to(DEV)


def lazy(t):
    """The values of t in a conjugated view."""
    v = t.conj().resolve_conj().conj()
    assert v.is_conj() and torch.equal(v, t)
    return v


STATE = [
    lambda s: ug.apply_operator(rand(2, 2, dtype=s.dtype), [1], s),
    lambda s: ug.apply_operator(rand(4, 4, dtype=s.dtype),
                                [np.int64(3), np.int64(0)], s),
    lambda s: ug.apply_operator(rand(3, 1, 2, 2, dtype=s.dtype), [1], s),
    lambda s: ug.apply_all_qubits(rand(2, 2, dtype=s.dtype), s),
    lambda s: ug.apply_each_qubit(rand(10, 2, 2, dtype=s.dtype), s),
    lambda s: ug.apply_phase(rand(1024).real.contiguous(), s),
    lambda s: ug.swap(s, (0, 3)),
    lambda s: ug.roll_qubits(s, 2),
    lambda s: ug.permute_qubits(list(range(10))[::-1], s),
    lambda s: ug.multi_cz(torch.tensor([[0, 1], [2, 5]], device=DEV), s),
    lambda s: ug.multi_controlled_x(s, [0, 1], 4),
    lambda s: simulation.multi_controlled_z([0, 1], s),
    lambda s: ug.norm_squared(s),
    lambda s: ug.abs_squared(s),
    lambda s: ug.inner_product(s, rand(1024, dtype=s.dtype)),
    lambda s: ug.inner_product(rand(1024, dtype=s.dtype), s),
    lambda s: ug.diag_expectation_value(
        torch.ones(1024, device=DEV, dtype=s.real.dtype), s),
    lambda s: states.norm_squared_fp64(s),
    lambda s: Circuit(10).h(0).cnot(0, 5).run(s),
    lambda s: measurement.sample(s[0, 0], 100, seed=1),
    lambda s: adjoint.pauli_expectation(adjoint.PauliSum(10).z(0), s),
]


@pytest.mark.parametrize("dtype", [C64, C128])
@pytest.mark.parametrize("call", range(len(STATE)))
def test_states(call, dtype):
    s = rand(3, 2, 1024, dtype=dtype)
    assert torch.equal(STATE[call](lazy(s)), STATE[call](s))


@pytest.mark.parametrize("dtype", [C64, C128])
@pytest.mark.parametrize("shape,qubits", [((2, 2), [1]),
                                          ((4, 4), [np.int64(2), 0]),
                                          ((3, 1, 2, 2), [0]),
                                          ((1, 1, 1, 2, 2), [0]),
                                          ((1, 1), [])])
def test_operators(shape, qubits, dtype):
    s, m = rand(3, 2, 1024, dtype=dtype), rand(*shape, dtype=dtype)
    assert torch.equal(ug.apply_operator(lazy(m), qubits, s),
                       ug.apply_operator(m, qubits, s))
    a, b = s.clone(), s.clone()
    simulation.apply_operator_(lazy(m), qubits, a)
    simulation.apply_operator_(m, qubits, b)
    assert torch.equal(a, b)
    if shape == (2, 2):
        assert torch.equal(ug.apply_all_qubits(lazy(m), s),
                           ug.apply_all_qubits(m, s))
        each = m.expand(10, 2, 2).contiguous()
        assert torch.equal(ug.apply_each_qubit(lazy(each), s),
                           ug.apply_each_qubit(each, s))


def test_in_place_on_a_lazy_view():
    s, m = rand(3, 1024), rand(2, 2)
    want = ug.apply_operator(m, [1], s)
    v = lazy(s)
    assert simulation.apply_operator_(m, [1], v) is v
    assert v.is_conj() and torch.equal(v, want)
    prog = Circuit(10).h(3).compile(C64, DEV)
    v = lazy(s)
    assert prog.run(v, inplace=True) is v
    assert torch.equal(v, prog.run(s))


def test_negated_angles():
    z = rand(1024)
    a = z.conj().imag  # a negated view
    assert a.is_neg()
    s = rand(3, 1024)
    assert torch.equal(ug.apply_phase(a, s),
                       ug.apply_phase(a.resolve_neg().contiguous(), s))


@pytest.mark.parametrize("dtype", [C64, C128])
def test_compiled_matrices(dtype):
    """Adjoints of gates (Circuit.inverse), on the host and on the device."""
    s = rand(2, 1024, dtype=dtype)
    c = Circuit(10).h(0).s(1).rx(2, 0.3)
    c.append(torch.linalg.qr(rand(8, 8, dtype=C128).cpu())[0], [3, 4, 5])
    eps = 1e-5 if dtype == C64 else 1e-12
    dev = Circuit(10)
    for g in c.inverse().gates:
        dev.append(lazy(g.matrix.resolve_conj().to(DEV)), g.qubits, g.kind)
    for back in (c.inverse(), dev):
        for fuse in (True, False):
            prog = back.compile(dtype, DEV, fuse=fuse)
            assert (prog.run(c.run(s)) - s).abs().max() < eps


GRAD = {
    "native": lambda m, e, a, s: ug.apply_operator(m, [1], s),
    "python": lambda m, e, a, s: ug.apply_operator(m, [np.int64(1)], s),
    "python, two": lambda m, e, a, s: ug.apply_operator(
        torch.kron(m, m), [np.int64(1), np.int64(4)], s),
    "broadcast": lambda m, e, a, s: ug.apply_operator(
        m.expand(3, 1, 2, 2), [1], s),
    "layer": lambda m, e, a, s: ug.apply_all_qubits(m, s),
    "layer, broadcast": lambda m, e, a, s: ug.apply_all_qubits(
        m.expand(3, 1, 2, 2), s),
    "each, broadcast": lambda m, e, a, s: ug.apply_each_qubit(
        e.expand(3, 1, 10, 2, 2), s),
    "phase": lambda m, e, a, s: ug.apply_phase(a, s),
    "phase, python": lambda m, e, a, s: ug.apply_phase(
        a.to(torch.float16), s),
}


@pytest.mark.parametrize("dtype", [C64, C128])
@pytest.mark.parametrize("name", GRAD)
def test_gradients(name, dtype):
    """d/dx of Re sum(conj(out) w): autograd's gradient of out is conj(w),
    lazily; the same loss as Re sum(out conj(w)) delivers it resolved."""
    w = rand(3, 2, 1024, dtype=dtype, seed=5)
    got = []
    for loss in (lambda o: (o.conj() * w).sum().real,
                 lambda o: (o * w.conj().resolve_conj()).sum().real):
        leaves = [t.requires_grad_() for t in (
            rand(2, 2, dtype=dtype), rand(10, 2, 2, dtype=dtype),
            rand(1024, dtype=dtype).real.contiguous(),
            rand(3, 2, 1024, dtype=dtype, seed=1))]
        out = GRAD[name](*leaves)
        got.append(torch.autograd.grad(loss(out), leaves, allow_unused=True))
    eps = 1e-5 if dtype == C64 else 1e-12
    assert any(g is not None for g in got[0])
    for a, b in zip(*got):
        assert (a is None) == (b is None)
        if a is not None:
            assert (a - b).abs().max() <= eps * b.abs().max()
