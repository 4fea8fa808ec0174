"""Tensor-core stages at the edges of their two kernels: one block up to more
than keep their images in shared memory (8), and tiles that leave groups,
buffers or whole SMs without work.

12 qubits are one tile, so a circuit of random 5-qubit unitaries is one stage
with about a block per gate.  Tolerance: the fp16 halves of the split are
rounded to 2^-12 of at most 1/2 in units where the column's largest amplitude
is at least 2^9 and the matrix's 2^10 at most; 64 products of both signs stay
below 64 * 2^-13 * 2^10 / (2^9 * 2^10) = 2^-16 of that amplitude in the worst
case, about an eighth of it (their root mean square) in practice, which is
2^-19 a block for a state of norm 1."""
import ctypes

import numpy as np
import pytest
import torch

from qcware_unitair_gb300 import _lib
from qcware_unitair_gb300.circuits import random_states
from qcware_unitair_gb300.fusion import Circuit

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _status():
    st = ctypes.c_int(-1)
    _lib.check(_lib.load().gbsv_tc_status(ctypes.byref(st), 1), "tc_status")
    return st.value


def _circuit(n, gates, seed):
    rng = np.random.default_rng(seed)
    circ = Circuit(n)
    for _ in range(gates):
        a = rng.normal(size=(32, 32)) + 1j * rng.normal(size=(32, 32))
        qs = [int(q) for q in rng.choice(n, size=5, replace=False)]
        circ.append(torch.from_numpy(np.linalg.qr(a)[0]), qs)
        # a diagonal between blocks
        d = np.diag(np.exp(1j * rng.uniform(0, 6.3, size=4)))
        qs = [int(q) for q in rng.choice(n, size=2, replace=False)]
        circ.append(torch.from_numpy(d), qs, "diag")
    return circ


@pytest.mark.parametrize("gates", [1, 2, 3, 4, 5, 6, 7, 8, 9, 12])
@pytest.mark.parametrize("n,batch", [(12, 1), (12, 2), (12, 460), (13, 2),
                                     (14, 229)])
def test_tc_stage_block_counts(oracle, n, batch, gates):
    _status()
    circ = _circuit(n, gates, 10 * n + gates)
    prog = circ.compile(torch.complex64, DEV, tensor_cores=True)
    assert prog.tensor_cores
    psi = random_states(n, (batch,), torch.complex64, seed=gates)
    out = prog.run(psi.to(DEV))
    some = sorted({0, 1, batch // 2, batch - 1} & set(range(batch)))
    ref = oracle.run_circuit(
        [(g.matrix.detach().cpu().numpy(), g.qubits) for g in circ.gates],
        psi[some].numpy().astype(np.complex128))
    err = np.abs(out[some].cpu().numpy() - ref).max()
    assert err <= 2.0 ** -19 * gates
    # every state of the batch: norms stay
    assert float((torch.linalg.vector_norm(out.to(torch.complex128), dim=-1)
                  - 1).abs().max()) <= 2.0 ** -19 * gates
    again = psi.to(DEV).clone()
    prog.run(again, inplace=True)
    assert torch.equal(again, out)
    assert _status() == 0
