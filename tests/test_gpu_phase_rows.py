"""apply_phase over broadcast rows and its backward, against complex128 torch:
rows below, at and above a block of columns, several rows per block, angles
shared or per row, states shared, every dtype pair.

Tolerance: the factor is rounded to the angle's precision (an error of at
most 2 ulp per component), the product to the output's: 8 * eps of the
largest amplitude for the coarser of the two; sums over broadcast rows add
one rounding per row."""
import numpy as np
import pytest
import torch

import qcware_unitair_gb300 as ug

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("shape_a,shape_s", [
    ((255,), (3, 255)), ((256,), (3, 256)), ((1024,), (9, 1024)),
    ((1025,), (1300, 1025)), ((5, 1), (5, 2048)), ((4, 1, 700), (1, 3, 700)),
    ((6, 512), (512,)), ((2, 1, 64), (2, 5, 64)), ((3, 300), (3, 300)),
    ((1,), (2, 1000)), ((7,), (2, 7))])
@pytest.mark.parametrize("da", [torch.float32, torch.float64])
@pytest.mark.parametrize("ds", [torch.complex64, torch.complex128])
def test_phase_and_gradients(shape_a, shape_s, da, ds):
    rng = np.random.default_rng(len(shape_a) + shape_s[-1])
    a = torch.from_numpy(rng.uniform(-9, 9, shape_a)).to(da).to(DEV)
    s = torch.from_numpy(rng.normal(size=shape_s) +
                         1j * rng.normal(size=shape_s)).to(ds).to(DEV)
    a.requires_grad_()
    s.requires_grad_()
    out = ug.apply_phase(a, s)
    w = torch.from_numpy(rng.normal(size=out.shape) + 1j *
                         rng.normal(size=out.shape)).to(out.dtype).to(DEV)
    out.backward(w)
    a2 = a.detach().double().requires_grad_()
    s2 = s.detach().to(torch.complex128).requires_grad_()
    ref = torch.exp(-1j * a2) * s2
    ref.backward(w.to(torch.complex128))
    assert out.dtype == torch.promote_types(
        ds, torch.complex64 if da == torch.float32 else torch.complex128)
    coarse = da == torch.float32 or ds == torch.complex64
    eps = 2.0 ** -24 if coarse else 2.0 ** -46
    for got, want in ((out, ref), (s.grad, s2.grad), (a.grad, a2.grad)):
        rows = max(1, out.numel() // got.numel())
        assert got.shape == want.shape
        off = (got.detach().to(want.dtype) - want.detach()).abs().max()
        # both factors of dL/da are up to |w| |out|
        size = want.detach().abs().max() + w.abs().max() * s.abs().max()
        assert off <= 8 * eps * rows * size


def test_second_derivative_of_the_angles():
    """d2/da2 of sum_k d_k |(U exp(-i a) psi)_k|^2 through create_graph: the
    angles' gradient stays differentiable."""
    rng = np.random.default_rng(5)
    n = 16
    a = torch.from_numpy(rng.uniform(-2, 2, n)).to(DEV).requires_grad_()
    psi = torch.from_numpy(rng.normal(size=n) + 1j * rng.normal(size=n)).to(
        DEV)
    u = torch.from_numpy(np.linalg.qr(rng.normal(size=(n, n)) + 1j *
                                      rng.normal(size=(n, n)))[0]).to(DEV)
    d = torch.from_numpy(rng.normal(size=n)).to(DEV)

    def energy(x, phase):
        out = u @ phase(x, psi)
        return (d * (out.conj() * out).real).sum()

    got, ref = [], []
    for phase, into in ((ug.apply_phase, got),
                        (lambda x, s: torch.exp(-1j * x) * s, ref)):
        g, = torch.autograd.grad(energy(a, phase), a, create_graph=True)
        into.append(torch.autograd.grad(g[3], a)[0])
    assert (got[0] - ref[0]).abs().max() <= 1e-12 * n * n


@pytest.mark.parametrize("cols", [2, 254, 1022, 1024, 1026, 4096])
@pytest.mark.parametrize("per_row", [False, True])
def test_pairs_equal_single_amplitudes(cols, per_row):
    """Two amplitudes at a time where every row is 16-byte aligned; the same
    data one amplitude off takes the other form and gives the same bits."""
    rng = np.random.default_rng(cols)
    rows = 9
    a = torch.from_numpy(rng.uniform(-9, 9, (rows, cols) if per_row else cols)
                         ).float().to(DEV)
    store = torch.zeros(rows * cols + 2, dtype=torch.complex64, device=DEV)
    off = store[1:1 + rows * cols].view(rows, cols)
    off.copy_(torch.from_numpy(rng.normal(size=(rows, cols)) +
                               1j * rng.normal(size=(rows, cols))))
    even = off.clone()
    assert torch.equal(ug.apply_phase(a, even), ug.apply_phase(a, off))
    # rows an odd number of amplitudes apart
    wide = torch.zeros(rows, cols + 1, dtype=torch.complex64, device=DEV)
    wide[:, :cols] = even
    assert torch.equal(ug.apply_phase(a, wide[:, :cols]),
                       ug.apply_phase(a, even))


@pytest.mark.parametrize("rows,cols", [(304, 1024), (305, 1024), (613, 512),
                                       (97, 4098), (330, 1026), (80, 4097)])
def test_rows_and_elements_agree(rows, cols):
    """Around 2048 elements per SM, where rows take over from elements: the
    forms give the same bits forward, and gradients within a rounding."""
    rng = np.random.default_rng(rows)
    a = torch.from_numpy(rng.uniform(-9, 9, cols)).float().to(DEV)
    s = torch.from_numpy(rng.normal(size=(rows, cols)) +
                         1j * rng.normal(size=(rows, cols))
                         ).to(torch.complex64).to(DEV)
    whole = ug.apply_phase(a, s)
    parts = torch.cat([ug.apply_phase(a, s[i:i + 8])
                       for i in range(0, rows, 8)])
    assert torch.equal(whole, parts)
    w = torch.from_numpy(rng.normal(size=(rows, cols)) + 0j
                         ).to(torch.complex64).to(DEV)
    grads = []
    for step in (rows, 8):
        x = s.clone().requires_grad_()
        t = a.expand(rows, cols).clone().requires_grad_()
        for i in range(0, rows, step):
            ug.apply_phase(t[i:i + step], x[i:i + step]).backward(
                w[i:i + step])
        grads.append((x.grad, t.grad))
    for g, h in zip(*grads):
        assert torch.equal(g, h)
