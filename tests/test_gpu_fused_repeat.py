"""complex128 register stages give the same bits whatever ran before them:
the choice between float pairs and FP64 must rest on the stage's own values,
not on what an earlier kernel left in shared memory."""
import pytest
import torch

import qcware_unitair_gb300 as ug
from qcware_unitair_gb300.circuits import random_circuit, random_states
from qcware_unitair_gb300.fusion import Circuit

pytestmark = pytest.mark.gpu


def fill_shared_memory(value):
    """A 5-qubit complex64 operator on 22 qubits keeps 139 KB per SM, all of
    it matrix and amplitudes; float patterns of 1e30 or infinity read as
    doubles beyond the pairs' range."""
    op = torch.full((32, 32), value, dtype=torch.complex64, device="cuda")
    state = torch.full((2 ** 22,), value, dtype=torch.complex64,
                       device="cuda")
    ug.apply_operator(op, [0, 3, 9, 17, 21], state)


@pytest.mark.parametrize("n,tile", [(14, 8), (16, 10), (16, 12)])
def test_same_bits(n, tile):
    circ = Circuit.from_gates(n, random_circuit(n, 300, seed=n + tile))
    for q in range(n):  # one-qubit diagonals: two values in a four-value slot
        circ.rz(q, 0.1 * (q + 1))
    prog = circ.compile(torch.complex128, "cuda", tile_qubits=tile)
    psi = random_states(n, (4,), torch.complex128, seed=n).cuda()
    fill_shared_memory(0j)
    want = prog.run(psi)
    for _ in range(5):
        fill_shared_memory(1e30 + 1e30j)
        assert torch.equal(prog.run(psi), want)
