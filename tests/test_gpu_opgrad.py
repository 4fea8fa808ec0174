"""Operator gradients (csrc/grad.cu) against complex128 torch einsum, at one
group, fewer groups than a block has threads, one and several parts, every
row split (k = 1..4), the general kernel (k = 5) and both directions at once
(k = 1, 2) or apart.

Tolerance: the gradient's sums are exact to about twice the precision, the
inputs of this call are exact, so what is left is the rounding of the result
(2^-24 relative for complex64) and of the state's gradient (2^k terms, each
product and sum rounded: at most 2^(k+2) roundings of the largest term)."""
import numpy as np
import pytest
import torch

import qcware_unitair_gb300 as ug

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _reference(m, qs, psi, g, n, shared):
    """(dL/dU, dL/dpsi) in complex128 for out = U psi, grad_out g."""
    k = len(qs)
    B = g.shape[0]

    def split(t):
        t = t.to(torch.complex128).expand(B, -1).reshape([B] + [2] * n)
        rest = [q for q in range(n) if q not in qs]
        t = t.permute([0] + [1 + q for q in qs] + [1 + q for q in rest])
        return t.reshape(B, 2 ** k, -1)

    gs, ps = split(g), split(psi)
    gu = torch.einsum("bar,bcr->bac", gs, ps.conj())
    m = m.to(torch.complex128)
    gp = torch.matmul(m.conj().transpose(-1, -2), gs)
    rest = [q for q in range(n) if q not in qs]
    order = [0] + [1 + q for q in list(qs) + rest]
    back = [order.index(i) for i in range(n + 1)]
    gp = gp.reshape([B] + [2] * n).permute(back).reshape(B, -1)
    return (gu.sum(0) if shared else gu), gp


@pytest.mark.parametrize("k,n,batch", [
    (1, 1, 3), (1, 6, 1), (1, 10, 5), (1, 17, 2), (2, 2, 1), (2, 9, 7),
    (2, 16, 3), (3, 3, 2), (3, 11, 5), (3, 15, 1), (4, 4, 1), (4, 13, 3),
    (5, 11, 2)])
@pytest.mark.parametrize("form", ["shared", "per_state", "broadcast_state",
                                  "operator_only"])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_operator_gradient(k, n, batch, form, dtype):
    rng = np.random.default_rng(100 * k + n)

    def rand(*shape):
        a = rng.normal(size=shape) + 1j * rng.normal(size=shape)
        return torch.from_numpy(a).to(dtype).to(DEV)

    d = 2 ** k
    per = form in ("per_state", "broadcast_state")
    m = rand(*((batch,) if per else ()), d, d)
    psi = rand(2 ** n) if form == "broadcast_state" else rand(batch, 2 ** n)
    w = rand(batch, 2 ** n)
    qs = [int(q) for q in rng.choice(n, size=k, replace=False)]
    m.requires_grad_()
    psi.requires_grad_(form != "operator_only")
    ug.apply_operator(m, qs, psi).backward(w)
    gu, gp = _reference(m.detach(), qs, psi.detach(), w, n, not per)
    eps = 2.0 ** -24 if dtype == torch.complex64 else 2.0 ** -46
    # complex128 sums in FP64: a sum of N terms rounds N times
    terms = 1 if dtype == torch.complex64 else 2.0 ** -7 * batch * 2 ** (n - k)
    scale = torch.linalg.vector_norm(gu)
    off = torch.linalg.vector_norm(m.grad.to(gu.dtype) - gu)
    assert off <= 2 * eps * max(1.0, terms) * scale
    if form == "operator_only":
        assert psi.grad is None
        return
    if form == "broadcast_state":
        gp = gp.sum(0)
    off = (psi.grad.to(gp.dtype) - gp).abs().max()
    assert off <= 4 * d * eps * gp.abs().max() * (
        batch if form == "broadcast_state" else 1)
