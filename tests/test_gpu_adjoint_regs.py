"""Register-layout backward stages against one kernel per gate
(_backward_sweep): every kind of op in every place (register, thread-index
and outside bits), more rotations than a CTA buffers, parameters that drive
several rotations, the smallest and largest tiles and the sizes below them.

Tolerance: both walk the same states with different rounding; per gate an
amplitude moves by a few eps, so G gates give G * 8 eps of the gradients'
scale (the norm of H, here at most the number of its terms)."""
import numpy as np
import pytest
import torch

from qcware_unitair_gb300 import adjoint as ad
from qcware_unitair_gb300.circuits import gate_matrix, random_states

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _circuit(n, gates, rng, shared):
    pc = ad.ParamCircuit(n, 5 if shared else gates)
    count = 0
    for _ in range(gates):
        kind = rng.choice(["rx", "ry", "rz", "rz", "h", "s", "t", "z", "cz",
                           "cnot", "swap", "u2"])
        q = [int(x) for x in rng.choice(n, size=2, replace=False)]
        if kind in ("rx", "ry", "rz"):
            p = count % 5 if shared else count
            getattr(pc, kind)(q[0], p, float(rng.choice([1.0, -0.5, 2.0])))
            count += 1
        elif kind == "u2":
            a = rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4))
            pc.gate(np.linalg.qr(a)[0], q)
        elif kind in ("h", "s", "t", "z"):
            pc.gate(gate_matrix(kind.upper()), q[:1],
                    "dense" if kind == "h" else "diag")
        else:
            pc.gate(gate_matrix(kind.upper()), q,
                    {"cz": "diag", "cnot": "ctrl"}.get(kind, "dense"))
    return pc


@pytest.mark.parametrize("n,batch,gates", [(7, 2, 60), (8, 3, 60),
                                           (9, 3, 150), (11, 2, 80),
                                           (12, 1, 80), (13, 3, 90),
                                           (16, 2, 120)])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("shared", [False, True])
def test_register_stages_match_gate_by_gate(n, batch, gates, dtype, shared):
    rng = np.random.default_rng(n * gates)
    pc = _circuit(n, gates, rng, shared)
    H = ad.PauliSum(n)
    for q in range(n):
        H.z(q, float(rng.uniform(-1, 1)))
    H.xx(0, n - 1, 0.7)
    real = torch.float32 if dtype == torch.complex64 else torch.float64
    params = torch.from_numpy(rng.normal(size=(batch, pc.num_params))).to(
        real).to(DEV)
    psi0 = random_states(n, (batch,), dtype, seed=n).to(DEV)
    psi_L, _ = ad._forward(pc, params, dtype, psi0, False)
    got = ad._backward_fused(pc, params, H, psi_L, [], dtype)
    ref = ad._backward_sweep(pc, params, H, psi_L, [], dtype)
    eps = 2.0 ** -24 if dtype == torch.complex64 else 2.0 ** -47
    per = gates if shared else 1  # rotations that add into one gradient
    assert (got - ref).abs().max() <= 8 * eps * gates * (n + 1) * per


def test_register_stage_sums_more_slots_than_fit_at_once(monkeypatch):
    n, batch = 14, 2
    pc = ad.hardware_efficient_ansatz(n, 4)
    rng = np.random.default_rng(1)
    params = torch.from_numpy(rng.normal(size=(batch, pc.num_params))).to(
        torch.float32).to(DEV)
    H = ad.PauliSum(n).z(0).xx(2, 5, 0.3)
    psi_L, saved = ad._forward(pc, params, torch.complex64, None, True)
    ref = ad._backward_fused(pc, params, H, psi_L, saved, torch.complex64)
    monkeypatch.setattr(ad, "_PARTIAL_BYTES", 0)  # one stage at a time
    got = ad._backward_fused(pc, params, H, psi_L, saved, torch.complex64)
    assert torch.equal(got, ref)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,layers,checkpoints", [(3, 1, True), (9, 5, True),
                                                  (13, 4, True),
                                                  (13, 4, False)])
def test_sweep_in_its_own_states_equals_the_copying_one(n, layers, checkpoints,
                                                        dtype):
    """The public call lets the sweep run in the forward pass's own states;
    the same kernels on copies give the same bits, also with a psi0, which
    keeps the copies."""
    B = 3
    pc = ad.hardware_efficient_ansatz(n, layers)
    if layers == 5:  # a gate outside the stages
        a = np.random.default_rng(n).normal(size=(8, 8))
        pc.gate(torch.from_numpy(np.linalg.qr(a)[0] + 0j), [0, n // 2, n - 1])
    H = ad.PauliSum(n).z(0).xx(0, n - 1, 0.5)
    g = torch.Generator().manual_seed(n)
    params = torch.randn(B, pc.num_params, generator=g,
                         dtype=torch.float64).to(DEV)
    psi_L, saved = ad._forward(pc, params, dtype, None, checkpoints)
    ref = ad._backward_fused(pc, params, H, psi_L, saved, dtype)
    vals, got = ad.expectation_and_grad(pc, params, H, dtype=dtype,
                                        checkpoints=checkpoints)
    assert torch.equal(got, ref)
    assert torch.equal(vals, ad.pauli_expectation(H, psi_L))
    p = params.clone().requires_grad_()
    out = ad.expectation(pc, p, H, dtype=dtype, checkpoints=checkpoints)
    assert torch.equal(out.detach(), vals)
    out.sum().backward()
    assert torch.equal(p.grad, ref)
    psi0 = torch.zeros(B, 2 ** n, dtype=dtype, device=DEV)
    psi0[:, 0] = 1
    _, again = ad.expectation_and_grad(pc, params, H, psi0=psi0, dtype=dtype,
                                       checkpoints=checkpoints)
    assert torch.equal(again, ref)
