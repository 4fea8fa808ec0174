"""Amplitudes that overflow on the way through a layer or its gradient, or
that enter a Pauli sum infinite: the same infinities and NaNs as gate by gate
(in the order of the qubits, which is the order inside a pass), or as the
terms' complex products.  Exact where not finite."""
import numpy as np
import pytest
import torch

import qcware_unitair_gb300 as ug

pytestmark = pytest.mark.gpu
DEV = "cuda"


def gate(name):
    t = torch.tensor(0.7)
    m = {"H": ug.gates.hadamard(), "RX": ug.gates.rx(t),
         "RY": ug.gates.ry(t), "RZ": ug.gates.rz(t),
         "full": ug.gates.rx(t) @ ug.gates.rz(t) @ ug.gates.ry(t),
         "2^25 H": ug.gates.hadamard() * 2.0 ** 25}[name]
    return m.to(torch.complex64).to(DEV)


def large(n, batch, seed):
    """Some components near FP32's largest, the others of order 1; the
    second state below 2^16, but not by much."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1, 1, size=(batch, 2 ** n, 2))
    x[:1][rng.random((1,) + x.shape[1:]) < 0.5] *= 3.4e38
    x[1:] *= 6e4
    return torch.from_numpy((x @ [1, 1j]).astype(np.complex64)).to(DEV)


def equal(got, want):
    a, b = torch.view_as_real(got), torch.view_as_real(want)
    assert torch.equal(a.isnan(), b.isnan())
    assert torch.equal(a.nan_to_num(7.0), b.nan_to_num(7.0))


@pytest.mark.parametrize("n", [5, 9, 12, 14, 18, 21])
@pytest.mark.parametrize("name", ["H", "RX", "RY", "RZ", "full", "2^25 H"])
@pytest.mark.parametrize("in_place", [False, True])
def test_layers(n, name, in_place):
    m, psi = gate(name), large(n, 2, n)
    loop = psi
    for q in range(n):
        loop = ug.apply_operator(m, [q], loop)
    assert not loop[0].isfinite().all() or name == "RZ"
    if in_place:  # the C ABI's own in-place form
        from qcware_unitair_gb300 import _core, _lib
        out = psi.clone()
        _lib.check(_lib.load().gbsv_apply_all_qubits(
            out.data_ptr(), out.data_ptr(), _lib.C64, n, 2, 2 ** n,
            m.data_ptr(), 0, 0, _core.stream_of(out.device)), "layer")
        equal(out, loop)
        return
    equal(ug.apply_all_qubits(m, psi), loop)
    equal(ug.apply_each_qubit(m.expand(n, 2, 2).contiguous(), psi), loop)
    one = ug.apply_all_qubits(m.requires_grad_(), psi).detach()
    equal(one, loop)


@pytest.mark.parametrize("n,operator", [(9, True), (12, True), (9, False),
                                        (14, False)])
@pytest.mark.parametrize("name", ["H", "RX", "RZ", "full"])
def test_layer_state_gradients(n, operator, name):
    """A layer of adjoints from the first qubit, in the kernel that also
    gives the operator's gradient (one pass, up to 12 qubits) or alone."""
    m = gate(name).requires_grad_(operator)
    psi = large(n, 2, n).requires_grad_()
    w = large(n, 2, n + 1)
    got = torch.autograd.grad(ug.apply_all_qubits(m, psi), psi, w)[0]
    loop = w
    adj = m.detach().conj().T.resolve_conj().contiguous()
    for q in range(n):
        loop = ug.apply_operator(adj, [q], loop)
    equal(got, loop)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n", [1, 2, 3, 8, 13])
def test_pauli_sums(n, dtype):
    """A real coefficient is multiplied as the complex number it is: an
    infinite partner gives NaN in the other component."""
    from qcware_unitair_gb300.adjoint import PauliSum, _pauli_apply
    rng = np.random.default_rng(n)
    psi = torch.from_numpy(rng.normal(size=(3, 2 ** n, 2)) @ [1, 1j]).to(
        dtype).to(DEV)
    psi[1, 1] = complex(float("inf"), 0.5)
    psi[2, 0] = complex(0.25, float("nan"))
    H = PauliSum(n).z(0).add(0.5, {0: "X"}).add(-2.0, {n - 1: "Y"}).z(
        n - 1, 0.3)
    got = _pauli_apply(H, psi, torch.empty_like(psi))
    x = np.arange(2 ** n)
    re, im = np.zeros((2, 3, 2 ** n))
    host = psi.cpu().numpy().astype(complex)
    for t in H.term_array():
        y = x ^ int(t["x"])
        sign = 1 - 2 * (np.array([bin(v & int(t["z"])).count("1")
                                  for v in y]) & 1)
        a, b = host[:, y].real * sign, host[:, y].imag * sign
        with np.errstate(invalid="ignore"):
            re, im = (re + (t["re"] * a - t["im"] * b),
                      im + (t["re"] * b + t["im"] * a))
    eps = 1e-5 if dtype == torch.complex64 else 1e-13
    for g, w in ((got.real, re), (got.imag, im)):
        g = g.cpu().numpy().astype(float)
        assert np.array_equal(np.isnan(g), np.isnan(w))
        fin = np.isfinite(w)
        assert np.array_equal(g[~fin & ~np.isnan(w)], w[~fin & ~np.isnan(w)])
        assert np.abs(g[fin] - w[fin]).max(initial=0) < eps
