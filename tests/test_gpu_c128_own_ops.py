"""complex128 2x2 operators of their own for each state: the forms that leave
out products with zeros, states with different forms in one warp, and
amplitudes that are not finite, where the full product is kept.

Tolerance: FP64, four products per component: 8 * 2^-53 of the largest
amplitude.  A non-finite amplitude gives NaN in exactly the components where
the full products do."""
import numpy as np
import pytest
import torch

import qcware_unitair_gb300 as ug
from qcware_unitair_gb300.circuits import gate_matrix

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _ops(kinds, rng):
    out = []
    for k in kinds:
        if k == "U":
            a = rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2))
            out.append(np.linalg.qr(a)[0])
        else:
            out.append(gate_matrix(k, float(rng.uniform(0, 6))))
    return np.stack(out).astype(np.complex128)


@pytest.mark.parametrize("n", [1, 2, 3, 6, 9])
@pytest.mark.parametrize("kinds", [("RX",), ("RY",), ("RZ",), ("U",),
                                   ("RX", "RY", "RZ", "U")])
def test_own_operators(oracle, n, kinds):
    rng = np.random.default_rng(n)
    batch = 13
    m = _ops([kinds[i % len(kinds)] for i in range(batch)], rng)
    psi = rng.normal(size=(batch, 2 ** n)) + 1j * rng.normal(
        size=(batch, 2 ** n))
    for q in sorted({0, n // 2, n - 1}):
        got = ug.apply_operator(torch.from_numpy(m).to(DEV), [q],
                                torch.from_numpy(psi).to(DEV)).cpu().numpy()
        ref = np.stack([oracle.run_circuit([(m[i], (q,))], psi[i:i + 1])[0]
                        for i in range(batch)])
        assert np.abs(got - ref).max() <= 8 * 2.0 ** -53 * np.abs(psi).max()


@pytest.mark.parametrize("kind", ["RX", "RY", "RZ"])
def test_not_finite(kind):
    rng = np.random.default_rng(1)
    m = torch.from_numpy(_ops([kind] * 4, rng)).to(DEV)
    psi = torch.ones(4, 64, dtype=torch.complex128, device=DEV)
    psi[1, 5] = complex(float("inf"), 0.0)
    out = ug.apply_operator(m, [5], psi).cpu().numpy()
    # every product of the pair (4, 5), those with zeros too
    a, e = psi[1, 4:6].cpu().numpy(), m[1].cpu().numpy()
    with np.errstate(invalid="ignore"):
        re = [sum(e[r, c].real * a[c].real - e[r, c].imag * a[c].imag
                  for c in (0, 1)) for r in (0, 1)]
        im = [sum(e[r, c].real * a[c].imag + e[r, c].imag * a[c].real
                  for c in (0, 1)) for r in (0, 1)]
    assert np.array_equal(np.isnan(out.real[1, 4:6]), np.isnan(re))
    assert np.array_equal(np.isnan(out.imag[1, 4:6]), np.isnan(im))
    assert np.isnan(re).any() or np.isnan(im).any()
    out[1, 4:6] = 0
    assert np.isfinite(out.real).all() and np.isfinite(out.imag).all()
