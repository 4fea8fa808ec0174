"""An operator that is changed in place between forward and backward: the
state's gradient (and a layer's operator gradient) needs the values of the
forward pass, so backward raises, as torch's own functions do.  Where only
the operator's gradient is asked for the operator is not needed, and where
its batch was expanded the node holds a copy: then the gradients are those of
the forward pass."""
import numpy as np
import pytest
import torch

import qcware_unitair_gb300 as ug

pytestmark = pytest.mark.gpu
DEV = "cuda"
N = 10


def operator(*batch):
    g = torch.Generator().manual_seed(1)
    return torch.randn(*batch, 2, 2, dtype=torch.complex64,
                       generator=g).to(DEV)


def state(*batch):
    g = torch.Generator().manual_seed(2)
    return torch.randn(*batch, 2 ** N, dtype=torch.complex64,
                       generator=g).to(DEV)


CALLS = {
    "gate": (lambda m, s: ug.apply_operator(m, [1], s), (), True),
    "gate, python": (lambda m, s: ug.apply_operator(m, [np.int64(1)], s), (),
                     True),
    "gate, batch": (lambda m, s: ug.apply_operator(m, [1], s), (3, 1), True),
    "layer": (ug.apply_all_qubits, (), False),
    "layer, batch": (ug.apply_all_qubits, (3, 1), False),
    "each": (ug.apply_each_qubit, (N,), False),
    "each, batch": (ug.apply_each_qubit, (3, 1, N), False),
}


@pytest.mark.parametrize("name", CALLS)
def test_changed_in_place(name):
    call, batch, gate = CALLS[name]
    for op_grad, state_grad in ((False, True), (True, True), (True, False)):
        got = []
        for change in (False, True):
            m = operator(*batch).requires_grad_(op_grad)
            s = state(3, 2).requires_grad_(state_grad)
            op = m * 1  # not a leaf, so that it may be changed in place
            out = call(op, s).abs().sum()
            if change:
                with torch.no_grad():
                    op.mul_(2)
            wrt = [t for t in (m, s) if t.requires_grad]
            if change and len(batch) < 2 and not (gate and not state_grad):
                with pytest.raises(RuntimeError, match="inplace operation"):
                    torch.autograd.grad(out, wrt)
            else:
                got.append(torch.autograd.grad(out, wrt))
        for a, b in zip(got[0], got[-1]):
            assert torch.equal(a, b)


@pytest.mark.parametrize("name", CALLS)
def test_hooks_see_the_operator(name):
    call, batch, _ = CALLS[name]
    m = operator(*batch).requires_grad_()
    s = state(3, 2).requires_grad_()
    packed = []

    def pack(t):
        packed.append(t.detach().clone())
        return t

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        out = call(m, s)
    shapes = [t.numel() for t in packed]
    assert any(n in (m.numel(), 6 * m.numel() // 3) for n in shapes)
    want = torch.autograd.grad(call(m, s).abs().sum(), (m, s))
    got = torch.autograd.grad(out.abs().sum(), (m, s))
    for a, b in zip(got, want):
        assert torch.equal(a, b)
