"""Tensor-core stages of gates that are not unitary: scaled unitaries,
imaginary-time steps, projectors and damping.

Block matrices then leave the range of an fp16 image (entries up to 2, rows'
L1 norm up to 8, columns not far below 1), so they are stored divided by a
power of two per column, which the kernel multiplies the amplitudes by.
Executed from the records on the CPU, and on the GPU (both stage kernels).

Tolerance: an image keeps 2^-22 of a column's largest entry, blocks add up
like independent errors, so sqrt(16) * 2^-22 * 2 = 2e-6 of the state's norm
for the up to 16 blocks here, and three times that for the 35 on the GPU with
the rounding of the amplitudes' split; the register stages' own error, which
is larger where a step amplifies, is allowed on top there."""
import numpy as np
import pytest
import torch

import test_tc_exec as exec_
from oracle import oracle as O
from qcware_unitair_gb300 import tcplan
from qcware_unitair_gb300.circuits import random_circuit
from qcware_unitair_gb300.fusion import Circuit

BOUND = 2e-6


def scaled(n, gates, factor, seed=1):
    return [(factor * g.matrix(), list(g.qubits))
            for g in random_circuit(n, gates, seed=seed)]


def imaginary_time(n, steps, tau):
    x = np.cosh(tau) * np.eye(2) + np.sinh(tau) * np.array([[0, 1], [1, 0]])
    zz = np.diag(np.exp(tau * np.array([1.0, -1, -1, 1])))
    step = [(zz, [q, q + 1]) for q in range(n - 1)] + [
        (x, [q]) for q in range(n)]
    return step * steps


def damped(n, gates, small):
    """Projectors, damping and jumps between random gates."""
    rng = np.random.default_rng(0)
    out = []
    for i, g in enumerate(random_circuit(n, gates, seed=2)):
        out.append((g.matrix(), list(g.qubits)))
        q = [int(rng.integers(n))]
        if i % 9 == 0:
            out.append((np.diag([1.0, 0.0]), q))
        if i % 7 == 0:
            out.append((np.diag([1.0, small]), q))
        if i % 11 == 0:
            out.append((np.array([[1.0, small], [0.0, 1e-3]]), q))
    return out


CASES = {
    "unitary": lambda n: scaled(n, 40, 1.0),
    "x0.7": lambda n: scaled(n, 120, 0.7),
    "x0.5": lambda n: scaled(n, 120, 0.5),
    "x1.5": lambda n: scaled(n, 120, 1.5),
    "imaginary time": lambda n: imaginary_time(n, 10, 0.5),
    "short steps": lambda n: imaginary_time(n, 10, 0.05),
    "damped 1e-4": lambda n: damped(n, 60, 1e-4),
    "damped 1e-7": lambda n: damped(n, 60, 1e-7),
}


def circuit(n, gates):
    c = Circuit(n)
    for m, q in gates:
        c.append(torch.from_numpy(np.asarray(m, np.complex128)), q)
    return c


def relative(got, want):
    return float((np.linalg.norm(got - want, axis=-1) /
                  np.linalg.norm(want, axis=-1)).max())


def run_records(prog, psi, monkeypatch):
    """exec_.run_tc_records with the column scales put into the matrices
    (scaling the amplitudes by powers of two is exact)."""
    blocks, diags, images, factors = prog.tc_records
    flat = np.concatenate(factors) if factors else np.zeros(0, np.complex64)
    matrices = []
    for blk in blocks:
        img = images[int(blk["mat"])]
        assert np.isfinite(img).all()
        high = img[tcplan._IMG_IDX[64:]].astype(np.float64)
        assert np.abs(high).max() <= 2048
        assert np.abs(high).sum(axis=0).max() <= 8.01 * 1024 + 32
        m = tcplan.image_matrix(img)
        if int(blk["flags"]) & tcplan.TC_COLS:
            at = int(blk["cols"])
            s = flat[at:at + 16].view(np.float32).astype(np.float64)
            assert np.all((s == 0) | (np.frexp(s)[0] == 0.5))
            m = np.repeat(s, 2)[:, None] * m
        matrices.append(m)

    class Records:
        n, ops = prog.n, prog.ops
        tc_records = (blocks, diags, matrices, factors)

    monkeypatch.setattr(tcplan, "image_matrix", lambda m: m)
    return exec_.run_tc_records(Records, psi)


@pytest.mark.parametrize("name", CASES)
def test_records(name, monkeypatch):
    n = 14
    gates = CASES[name](n)
    prog = circuit(n, gates).compile(device="cpu")
    assert prog.tensor_cores
    psi = exec_._states(n, 2, 0)
    got = run_records(prog, psi, monkeypatch)
    assert relative(got, O.run_circuit(gates, psi)) < BOUND


def test_unitaries_are_not_scaled():
    prog = Circuit.from_gates(14, random_circuit(14, 200, seed=3)).compile(
        device="cpu")
    assert not any(int(b["flags"]) & tcplan.TC_COLS
                   for b in prog.tc_records[0])
    flat = np.kron(np.kron([[1, 1j], [1j, 1]], [[1, 1], [1, -1]]),
                   np.ones((8, 8))) / 8
    for u in (flat, np.eye(32)):
        # entries as small as a unitary's can be
        assert tcplan.column_scales(u / np.abs(u).max() / 8)[0] is None


def test_column_scales():
    rng = np.random.default_rng(4)
    for shift in (-200, -40, -4, 4, 40):
        u = rng.normal(size=(32, 32)) + 1j * rng.normal(size=(32, 32))
        u = u * 2.0 ** (shift + rng.integers(-9, 9, size=32))
        u[:, 5] = 0
        s, w = tcplan.column_scales(u)
        assert s[5] == 0 and np.all(w[:, 5] == 0)
        assert np.array_equal(w * s, u)
        assert tcplan._row_l1(w) <= 8
        if shift > -200:  # beyond FP32's powers of two the entries stay small
            assert np.abs(w).max() > 1 / 16


@pytest.mark.gpu
@pytest.mark.parametrize("n", [12, 14])
@pytest.mark.parametrize("name", CASES)
def test_gpu(name, n):
    """12 qubits: one stage of all blocks (more than eight: the kernel that
    streams images); 14: several shorter ones."""
    gates = CASES[name](n)
    c = circuit(n, gates)
    psi = exec_._states(n, 3, 1)
    x = torch.from_numpy(psi.astype(np.complex64)).cuda()
    want = O.run_circuit(gates, x.cpu().numpy().astype(np.complex128))
    err = {}
    for tc in (True, False):
        out = c.compile(torch.complex64, "cuda", tensor_cores=tc).run(x)
        err[tc] = relative(out.cpu().numpy().astype(np.complex128), want)
    print(f"{name} n={n}: tensor cores {err[True]:.2e}, registers "
          f"{err[False]:.2e}")
    assert err[True] < 3 * BOUND + err[False]
