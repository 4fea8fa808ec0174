"""gbsv_plan_tc on long lists in which a qubit sees only diagonal gates: the
scans keep an early end (the time grows with the list, not with its square),
and the plan is still the circuit."""
import time

import numpy as np
import torch

import test_tc_exec as exec_
from oracle import oracle as O
from qcware_unitair_gb300 import _lib
from qcware_unitair_gb300.fusion import Circuit


def masks(n, gates, lone, seed=0):
    """Two-qubit gates on random positions; every other one diagonal and on
    position 0, which sees no others, where ``lone``."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(gates):
        if lone and i % 2:
            a, b = 0, 1 + int(rng.integers(n - 1))
        else:
            a, b = (1 + int(x) for x in rng.choice(n - 1, 2, replace=False))
        out.append((1 << a) | (1 << b))
    diag = [lone and i % 2 for i in range(gates)]
    return np.array(out, np.uint64), np.array(diag, np.uint8)


def seconds(lib_built, *args):
    m, d = masks(*args)
    stage, block = np.zeros((2, len(m)), np.int32)
    post = np.zeros(len(m), np.uint8)
    t = time.perf_counter()
    assert _lib.load().gbsv_plan_tc(
        m.ctypes.data, d.ctypes.data, len(m), 4, stage.ctypes.data,
        block.ctypes.data, post.ctypes.data) == 0
    return time.perf_counter() - t


def test_time_grows_with_the_list(lib_built):
    seconds(lib_built, 26, 100, True)
    short = min(seconds(lib_built, 26, 1500, True) for _ in range(3))
    # eight times the gates: 64 times the work where it is quadratic
    long = min(seconds(lib_built, 26, 12000, True) for _ in range(2))
    assert long < 30 * short + 0.1


def test_long_circuit_with_a_diagonal_qubit(lib_built):
    n, gates = 13, 700
    rng = np.random.default_rng(1)
    c, ref = Circuit(n), []
    for i in range(gates):
        if i % 2:
            q = [0, 1 + int(rng.integers(n - 1))]
            m = np.diag(np.exp(1j * rng.uniform(0, 6, 4)))
        else:
            q = [int(x) for x in 1 + rng.choice(n - 1, 2, replace=False)]
            a = rng.normal(size=(4, 4, 2)) @ [1, 1j]
            m = np.linalg.qr(a)[0]
        c.append(torch.from_numpy(m), q)
        ref.append((m, q))
    prog = c.compile(device="cpu", tensor_cores=True)
    psi = exec_._states(n, 1, 2)
    got = exec_.run_tc_records(prog, psi)
    # 2e-6 for 150-gate circuits (test_tc_exec), errors of blocks adding up
    # like independent ones
    assert np.abs(got - O.run_circuit(ref, psi)).max() < 2e-6 * 5 ** 0.5
