"""Small complex128 components beside large ones: the pair arithmetic keeps a
float's 24 bits of a component down to 2^-126, whatever the other amplitudes
of its thread are (components that far apart are not mixed by these gates).

Tolerance: a small component is split to 2^-25 of itself, and a row has up to
16 real products, each at most twice the groups' size: 16 * 2 * 2^-25 = 2^-20
of the size, which is 2^-16 of an output that is at least a sixteenth of it
(what cancels below 2^-126 becomes zero, and is not looked at).  Large
components: the engine's 1e-12."""
import numpy as np
import pytest
import torch

import qcware_unitair_gb300 as ug

pytestmark = pytest.mark.gpu


def gate(name, k, rng):
    h = np.array([[1, 1], [1, -1]]) / np.sqrt(2)
    x = np.array([[0, 1], [1, 0]])
    one = {"H": h, "RX": np.cos(0.3) * np.eye(2) - 1j * np.sin(0.3) * x,
           "RZ": np.diag(np.exp([-0.3j, 0.3j]))}
    if name == "full":
        a = rng.normal(size=(2 ** k, 2 ** k, 2)) @ [1, 1j]
        return np.linalg.qr(a)[0]
    m = np.eye(1)
    for _ in range(k):
        m = np.kron(m, one[name])
    return m


@pytest.mark.parametrize("name", ["H", "RX", "RZ", "full"])
@pytest.mark.parametrize("k", [1, 2, 3])
@pytest.mark.parametrize("n", [8, 15])
def test_components(n, k, name):
    rng = np.random.default_rng(n * 10 + k)
    m = gate(name, k, rng)
    qubits = [int(q) for q in rng.choice(n, k, replace=False)]
    groups = 2 ** (n - k)
    for e in (-50, -80, -100, -106, -112, -119, -121):
        # each group of amplitudes that the gate mixes: of order 1 or 2^e
        size = np.where(rng.random(groups) < 0.5, 1.0, 2.0 ** e)
        x = (rng.uniform(1, 2, (2 ** k, groups, 2)) *
             rng.choice([-1, 1], (2 ** k, groups, 2))) @ [1, 1j] * size
        want = m @ x
        axes = qubits + [q for q in range(n) if q not in qubits]
        state = np.ascontiguousarray(x.reshape((2,) * n).transpose(
            np.argsort(axes))).reshape(-1)
        out = ug.apply_operator(torch.from_numpy(m.astype(complex)).cuda(),
                                qubits, torch.from_numpy(state).cuda())
        got = out.cpu().numpy().reshape((2,) * n).transpose(axes).reshape(
            2 ** k, groups)
        assert np.abs(got - want)[:, size == 1].max() < 1e-12
        for part in ("real", "imag"):
            g, w = getattr(got, part), getattr(want, part)
            look = (np.abs(w) > size / 16) & (size != 1)
            assert np.abs(g / np.where(look, w, 1) - 1)[look].max() < \
                2.0 ** -16, e
