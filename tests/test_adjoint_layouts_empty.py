"""Backward layouts whose gates come to nothing (a diagonal of ones has no
sign to flip): the kernel takes a layout's last op as the one before its end,
so a layout without ops would look before the list."""
import ctypes

import numpy as np
import pytest
import torch

from qcware_unitair_gb300 import _lib
from qcware_unitair_gb300 import adjoint as ad


def layouts(pc, m, dtype):
    plan = ad._plan_backward_native(pc, 0, len(pc.ops), dtype,
                                    torch.device("cpu"), m, device_ops=False)
    code = _lib.C64 if dtype == torch.complex64 else _lib.C128
    out = []
    for kind, st in plan:
        rec = np.ascontiguousarray(st["records"])
        G = st["num_ops"]
        ops = np.empty(4 * G, ad.REGOP_DTYPE)
        lays = np.zeros(G, ad.LAYOUT_DTYPE)
        nops, count = ctypes.c_int(0), ctypes.c_int(0)
        _lib.check(_lib.load().gbsv_adjoint_layouts(
            rec.ctypes.data, G, m, 4 if code == _lib.C64 else 3,
            st["host_pool"].ctypes.data, code, ops.ctypes.data,
            ctypes.byref(nops), lays.ctypes.data, G, ctypes.byref(count)),
            "layouts")
        out.append((nops.value, lays[:count.value]))
    return out


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_no_layout_without_ops(lib_built, dtype):
    n = 10
    pc = ad.ParamCircuit(n, 4)
    for q in range(n):
        pc.gate(np.eye(4), [q, (q + 1) % n], "diag")
    for nops, lays in layouts(pc, n, dtype):
        assert nops == 0 and len(lays) == 0
    # between layouts that have some
    pc.h(0).rx(1, 0)
    for q in range(2, n):
        pc.h(q).gate(np.eye(2), [q], "diag")
    pc.gate(np.eye(2), [0], "diag")
    for nops, lays in layouts(pc, n, dtype):
        at = 0
        for lay in lays:
            assert lay["first"] == at and lay["count"] > 0
            at += lay["count"]
        assert at == nops > 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_gradients(dtype):
    n = 10
    pc = ad.ParamCircuit(n, 2)
    for q in range(n):
        pc.gate(np.eye(4), [q, (q + 1) % n], "diag")
    nothing = len(pc.ops)
    H = ad.PauliSum(n).z(0).xx(1, 2, 0.5)
    p = torch.tensor([[0.3, 0.7]], dtype=torch.float64, device="cuda")
    _, grads = ad.expectation_and_grad(pc, p, H, dtype=dtype)
    assert torch.equal(grads, torch.zeros_like(grads))
    pc.ry(0, 0).rx(1, 1)
    bare = ad.ParamCircuit(n, 2)
    bare.ops = pc.ops[nothing:]
    eps = 1e-5 if dtype == torch.complex64 else 1e-12
    for a, b in zip(ad.expectation_and_grad(pc, p, H, dtype=dtype),
                    ad.expectation_and_grad(bare, p, H, dtype=dtype)):
        assert (a - b).abs().max() < eps
