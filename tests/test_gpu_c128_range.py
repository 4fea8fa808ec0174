"""complex128 gates in pairs where a warp's amplitudes do or do not all lie in
[2^-40, 2^61): just inside, just outside, zeros and negative zeros among
them, and sums that cancel to exactly zero.

Tolerance: a pair drops less than 2^-48 of a component, an entry none and a
product or sum of four terms a few 2^-48; 2^-44 of the largest amplitude
covers a gate.  Where two equal products cancel the result is exactly 0."""
import numpy as np
import pytest
import torch

import qcware_unitair_gb300 as ug
from qcware_unitair_gb300.circuits import gate_matrix

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("gate", ["H", "RX", "RZ", "U"])
@pytest.mark.parametrize("low", [-39, -40, -41, -74, -75, None])
@pytest.mark.parametrize("qubit", [0, 6, 11])
def test_range_edges(oracle, gate, low, qubit):
    n = 12
    rng = np.random.default_rng(17)
    a = rng.normal(size=(8, 8)) + 1j * rng.normal(size=(8, 8))
    m = (np.linalg.qr(a[:2, :2])[0] if gate == "U" else
         gate_matrix(gate) if gate == "H" else gate_matrix(gate, 0.7))
    psi = rng.uniform(1, 2, (3, 2 ** n)) * rng.choice([-1, 1], (3, 2 ** n)) + \
        1j * rng.uniform(1, 2, (3, 2 ** n))
    some = rng.random(psi.shape) < 0.02
    small = 0.0 if low is None else 1.5 * 2.0 ** low
    psi.real[some] = small
    psi.imag[rng.random(psi.shape) < 0.02] = -small
    psi[1] *= 2.0 ** 60  # the top of the range; beyond it above 2^61
    psi[2] *= 2.0 ** -39
    got = ug.apply_operator(torch.from_numpy(m).to(DEV), [qubit],
                            torch.from_numpy(psi).to(DEV)).cpu().numpy()
    ref = oracle.run_circuit([(m, (qubit,))], psi)
    for r in range(3):
        assert np.abs(got[r] - ref[r]).max() <= 2.0 ** -44 * np.abs(psi[r]).max()


@pytest.mark.parametrize("n", [8, 14])
def test_cancelling_products_give_zero(n):
    h = ug.gates.hadamard(dtype=torch.complex128).to(DEV)
    psi = torch.full((2, 2 ** n), 0.3 - 0.7j, dtype=torch.complex128,
                     device=DEV)
    out = ug.apply_operator(h, [n - 1], psi)
    assert bool((out[:, 1::2] == 0).all())
