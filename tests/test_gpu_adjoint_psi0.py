"""A caller's psi0 is read, not written: the same call twice gives the same
answer, also where psi0 has the dtype and layout the engine runs in, and
changing psi0 between forward and backward does not reach the gradient."""
import numpy as np
import pytest
import torch

from qcware_unitair_gb300 import adjoint as ad
from qcware_unitair_gb300.circuits import random_states

pytestmark = pytest.mark.gpu
DEV = "cuda"


def case(n, layers, batch, ops=True):
    pc = ad.hardware_efficient_ansatz(n, layers) if ops else \
        ad.ParamCircuit(n, 3)
    g = torch.Generator().manual_seed(n)
    params = torch.randn(batch, pc.num_params, generator=g,
                         dtype=torch.float64).to(DEV)
    return pc, params, ad.PauliSum(n).z(0).xx(0, n - 1, 0.5)


FORMS = {
    "batch": lambda s: s,
    "one": lambda s: s[:1],
    "vector": lambda s: s[0],
    "strided": lambda s: torch.stack([s, s], -1)[..., 0],
    "conjugated": lambda s: s.conj(),
}


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("n,layers", [(5, 1), (5, 0), (10, 5), (13, 4)])
@pytest.mark.parametrize("checkpoints", [True, False])
def test_psi0_is_left_alone(n, layers, form, dtype, checkpoints):
    s = FORMS[form](random_states(n, (3,), dtype, seed=1).to(DEV))
    batch = 1 if form == "one" else 3
    pc, params, H = case(n, max(layers, 1), batch, ops=layers > 0)
    before = s.clone()
    want = None
    for fuse in (True, True, False):
        got = ad.expectation_and_grad(pc, params, H, psi0=s, dtype=dtype,
                                      checkpoints=checkpoints, fuse=fuse)
        assert torch.equal(s, before)
        if want is None:
            want = got
        for a, b in zip(got, want):
            if fuse:
                assert torch.equal(a, b)
            else:  # other kernels: the engine's tolerances
                eps = 1e-4 if dtype == torch.complex64 else 1e-11
                assert (a - b).abs().max() < eps
    p = params.clone().requires_grad_()
    value = ad.expectation(pc, p, H, psi0=s, dtype=dtype,
                           checkpoints=checkpoints)
    assert torch.equal(s, before)
    if layers:
        s.zero_()  # the forward pass is over
        value.sum().backward()
        assert torch.equal(value.detach(), want[0])
        assert torch.equal(p.grad, want[1])


def test_against_the_copying_sweep():
    n = 12
    pc, params, H = case(n, 4, 2)
    s = random_states(n, (2,), torch.complex64, seed=2).to(DEV)
    psi_L, saved = ad._forward(pc, params, torch.complex64, s, True)
    ref = ad._backward_fused(pc, params, H, psi_L, saved, torch.complex64)
    _, got = ad.expectation_and_grad(pc, params, H, psi0=s)
    assert torch.equal(got, ref)
