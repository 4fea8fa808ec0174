"""apply_phase over broadcast rows beyond the size at which rows take over
from elements (2048 elements per SM; 311,296 on 152): angles shared by the
rows and their own, states shared by rows of angles, rows in pairs of
amplitudes and alone (odd columns, states or row strides off a 16-byte
address), and the same backward.

Tolerance: the factor is rounded to float (at most 2 ulp per component), the
product to the output's: 8 * 2^-24 of the largest amplitude; a sum over
broadcast rows adds one rounding per row.  Pairs and single amplitudes give
the same bits."""
import ctypes

import numpy as np
import pytest
import torch

import qcware_unitair_gb300 as ug
from qcware_unitair_gb300 import _core, _lib

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
EPS = 2.0 ** -24


def make(shape_a, shape_s, odd=False, seed=0):
    rng = np.random.default_rng(seed + shape_s[-1])
    a = torch.from_numpy(rng.uniform(-9, 9, shape_a)).float().to(DEV)
    size = int(np.prod(shape_s))
    store = torch.zeros(size + 2, dtype=torch.complex64, device=DEV)
    s = store[1:1 + size] if odd else store[:size]
    s.copy_(torch.from_numpy(rng.normal(size=size) +
                             1j * rng.normal(size=size)))
    assert s.data_ptr() % 16 == (8 if odd else 0)
    return a, s.view(shape_s)


SHAPES = [
    ((1024,), (400, 1024)), ((1026,), (330, 1026)), ((1025,), (330, 1025)),
    ((256,), (1300, 256)), ((4096,), (77, 4096)), ((2 ** 16,), (5, 2 ** 16)),
    # angles of their own for each row
    ((400, 1), (400, 1024)), ((330, 1), (330, 1026)), ((330, 1), (330, 1025)),
    # one state under rows of angles, and under one angle each
    ((400, 1024), (1024,)), ((330, 1026), (1026,)), ((330, 1025), (1025,)),
    ((2000, 1), (512,)),
    # a batch on either side
    ((110, 1, 1026), (110, 3, 1026)), ((110, 1, 1026), (3, 1026)),
    ((1, 3, 1026), (110, 1, 1026)),
]


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("shape_a,shape_s", SHAPES)
def test_forward_and_gradients(shape_a, shape_s, odd):
    a, s = make(shape_a, shape_s, odd)
    a.requires_grad_()
    s.requires_grad_()
    out = ug.apply_phase(a, s)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert out.numel() > 2048 * sms
    rng = np.random.default_rng(1)
    w = torch.from_numpy(rng.normal(size=out.shape) + 1j *
                         rng.normal(size=out.shape)).to(out.dtype).to(DEV)
    got = torch.autograd.grad(out, (a, s), w)
    a2 = a.detach().double().requires_grad_()
    s2 = s.detach().to(torch.complex128).requires_grad_()
    ref = torch.exp(-1j * a2) * s2
    want = torch.autograd.grad(ref, (a2, s2), w.to(torch.complex128))
    for g, r in zip((out, *got), (ref, *want)):
        rows = max(1, out.numel() // g.numel())
        assert g.shape == r.shape
        off = (g.detach().to(r.dtype) - r.detach()).abs().max()
        size = r.detach().abs().max() + w.abs().max() * s.abs().max()
        assert off <= 8 * EPS * rows * size


@pytest.mark.parametrize("shape_a,shape_s", SHAPES)
def test_pairs_and_single_amplitudes(shape_a, shape_s):
    (a, s), (_, t) = make(shape_a, shape_s), make(shape_a, shape_s, True)
    assert torch.equal(ug.apply_phase(a, s), ug.apply_phase(a, t))


@pytest.mark.parametrize("cols,stride", [(1026, 1027), (1026, 1028),
                                         (1026, 1026), (1024, 1031)])
@pytest.mark.parametrize("own", [False, True])
def test_row_strides(cols, stride, own):
    """Rows further apart than they are long (the C ABI's descriptor): pairs
    only where every row is at a 16-byte address."""
    rows = 400
    rng = np.random.default_rng(cols)
    wide = torch.from_numpy((rng.normal(size=(rows, stride, 2)) @ [1, 1j])
                            .astype(np.complex64)).to(DEV)
    a = torch.from_numpy(rng.uniform(-9, 9, (rows, 1) if own else cols)
                         ).float().to(DEV)
    out = torch.empty(rows, cols, dtype=torch.complex64, device=DEV)
    d = _lib.Bcast()
    d.ndim = 2
    for i, (n, sa, sb) in enumerate(((rows, int(own), stride),
                                     (cols, int(not own), 1))):
        d.shape[i], d.stride_a[i], d.stride_b[i] = n, sa, sb
    _lib.check(_lib.load().gbsv_apply_phase(
        a.data_ptr(), _lib.F32, wide.data_ptr(), _lib.C64, out.data_ptr(),
        _lib.C64, ctypes.byref(d), _core.stream_of(DEV)), "apply_phase")
    assert torch.equal(out, ug.apply_phase(a, wide[:, :cols].contiguous()))
