"""Pauli sums by kind of term (diagonal, X strings, with Y or mixed), in any
order and number, on the smallest states and with unaligned buffers; and the
rotation matrices written into a program's pool.

Tolerance: each output sums T products of the state's precision, each rounded
once with a coefficient of at most 1: (T + 1) eps of the largest amplitude
times T."""
import numpy as np
import pytest
import torch

from qcware_unitair_gb300 import adjoint as ad
from qcware_unitair_gb300.circuits import random_states

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("n", [1, 2, 3, 7])
@pytest.mark.parametrize("count", [1, 2, 31, 256])
@pytest.mark.parametrize("letters", ["Z", "X", "Y", "XZ", "XYZ"])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("shift", [0, 1])
def test_pauli_sum_kinds(n, count, letters, dtype, shift):
    rng = np.random.default_rng(n * count)
    H = ad.PauliSum(n)
    for _ in range(count):
        k = int(rng.integers(1, n + 1))
        qs = rng.choice(n, size=k, replace=False)
        H.add(float(rng.uniform(-1, 1)),
              {int(q): str(rng.choice(list(letters))) for q in qs})
    psi = random_states(n, (3,), torch.complex128, seed=1).to(dtype)
    buf = torch.zeros(3 * 2 ** n + shift, dtype=dtype, device=DEV)
    x = buf[shift:].view(3, 2 ** n)
    x.copy_(psi)
    out = torch.empty_like(psi, device=DEV)
    ad._pauli_apply(H, x, out)
    ref = psi.to(torch.complex128).numpy() @ H.dense().T
    eps = 2.0 ** -24 if dtype == torch.complex64 else 2.0 ** -53
    assert np.abs(out.cpu().numpy() - ref).max() <= (
        4 * (count + 1) * eps * count * psi.abs().max().item())


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("real", [torch.float32, torch.float64,
                                  torch.float16])
def test_rotation_matrices(dtype, real):
    n, B = 4, 5
    pc = ad.ParamCircuit(n, 6)
    pc.rx(0, 0).ry(1, 1, -0.5).rz(2, 2).rx(3, 3, 2.0).rz(0, 4).ry(2, 5)
    g = torch.Generator().manual_seed(1)
    p = (torch.rand(B, 6, generator=g) * 9 - 4).to(real).to(DEV)
    prog, which, _ = ad._forward_program(pc, 0, len(pc.ops), B, dtype, DEV,
                                         True)
    ad._write_rotations(prog, which, ad._real_params(p))
    vals = ad._rotation_values(which, p, B, dtype)
    idx = torch.cat([torch.arange(off, off + B * nv, device=DEV)
                     for _, _, _, off, nv in which])
    eps = 2.0 ** -24 if dtype == torch.complex64 else 2.0 ** -52
    assert (prog.pool[idx] - vals).abs().max() <= 2 * eps
