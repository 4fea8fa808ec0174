"""Rotation gates of CUDA angles against the CPU builders (the torch
operations), values, gradients and second derivatives; strides, 0-d angles,
dtypes, a full last block and one more angle.

Tolerance: cos and sin agree to 2 ulp between the devices, a gradient adds
four products of them."""
import pytest
import torch

import qcware_unitair_gb300 as ug

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("gate", ["exp_x", "exp_y", "exp_z", "rx", "ry",
                                  "rz"])
@pytest.mark.parametrize("form", ["scalar", "one", "row", "column", "grid",
                                  "block", "more", "expanded"])
@pytest.mark.parametrize("real,dtype", [
    (torch.float32, torch.complex64), (torch.float64, torch.complex128),
    (torch.float64, torch.complex64), (torch.float32, torch.complex128),
    (torch.int64, torch.complex64)])
def test_rotations(gate, form, real, dtype):
    g = torch.Generator().manual_seed(3)
    base = (torch.rand(40, 7, generator=g, dtype=torch.float64) * 20 - 10)
    pick = {"scalar": lambda t: t[3, 2], "one": lambda t: t[2, 3:4],
            "row": lambda t: t[5], "column": lambda t: t[:, 4],
            "grid": lambda t: t[2:9:3, 1:6:2],
            "block": lambda t: t.reshape(-1)[:128],
            "more": lambda t: t.reshape(-1)[:129],
            "expanded": lambda t: t[1, 1].expand(5)}[form]
    fn = getattr(ug.gates, gate)
    eps = 2.0 ** -23 if torch.complex64 == dtype else 2.0 ** -52
    host = base.to(real)
    dev = host.to(DEV)
    grad = real.is_floating_point
    host.requires_grad_(grad)
    dev.requires_grad_(grad)
    want, got = fn(pick(host), dtype=dtype), fn(pick(dev), dtype=dtype)
    assert got.shape == want.shape and got.dtype == want.dtype
    assert (got.cpu() - want).abs().max() <= 4 * eps
    if not grad:
        return
    w = torch.randn(want.shape, generator=g, dtype=torch.complex128).to(dtype)
    first = []
    for m, a, ww in ((want, host, w), (got, dev, w.to(DEV))):
        loss = (ww.conj() * m).real.sum() + (m * m).real.sum()
        d, = torch.autograd.grad(loss, a, create_graph=True)
        d2, = torch.autograd.grad(d.square().sum(), a)
        d1, = torch.autograd.grad((ww.conj() * fn(pick(a), dtype=dtype))
                                  .real.sum(), a)
        first.append((d.detach().cpu(), d2.cpu(), d1.cpu()))
    for x, y in zip(*first):
        assert x.dtype == y.dtype
        # a gradient is rounded to the angles' type
        eps = max(eps, torch.finfo(x.dtype).eps)
        assert (x - y).abs().max() <= 64 * eps * max(1.0, x.abs().max())
