"""Calls that wait for the device let other Python threads run.  A stream
that is busy for a second with more launches behind it than its queue takes
makes a launch wait; a second thread must tick on meanwhile."""
import threading
import time

import pytest
import torch

import qcware_unitair_gb300 as ug

pytestmark = pytest.mark.gpu
DEV = "cuda"
BUSY, MOST = 1.0, 0.5  # seconds: the busy kernel, and between two ticks


def calls():
    s = torch.zeros(2 ** 8, dtype=torch.complex64, device=DEV)
    s[0] = 1
    op = torch.eye(2, dtype=torch.complex64, device=DEV)
    param = op.clone().requires_grad_()
    each = op.expand(8, 2, 2).contiguous()
    a = torch.zeros(2 ** 8, device=DEV)
    return {
        "gate": lambda: ug.apply_operator(op, [0], s),
        "gate with a gradient": lambda: ug.apply_operator(param, [0], s),
        "layer": lambda: ug.apply_all_qubits(op, s),
        "each": lambda: ug.apply_each_qubit(each, s),
        "phase": lambda: ug.apply_phase(a, s),
        "norm": lambda: ug.norm_squared(s),
        "abs": lambda: ug.abs_squared(s),
        "inner": lambda: ug.inner_product(s, s),
        "diagonal": lambda: ug.diag_expectation_value(a, s),
        "rotation": lambda: ug.gates.rx(a),
    }


@pytest.fixture(scope="module")
def cycles():
    """torch.cuda._sleep's argument for BUSY seconds."""
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    t = time.perf_counter()
    torch.cuda._sleep(20_000_000)
    torch.cuda.synchronize()
    return int(BUSY * 20_000_000 / (time.perf_counter() - t))


@pytest.mark.parametrize("name", [
    "gate", "gate with a gradient", "layer", "each", "phase", "norm", "abs",
    "inner", "diagonal", "rotation"])
def test_other_threads_run(name, cycles):
    call = calls()[name]
    call()
    torch.cuda.synchronize()
    gaps, stop = [], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    other = threading.Thread(target=tick)
    other.start()
    torch.cuda._sleep(cycles)
    start = time.perf_counter()
    for _ in range(3000):
        call()
    waited = time.perf_counter() - start
    stop.set()
    other.join()
    torch.cuda.synchronize()
    assert waited > BUSY / 2  # the queue was full, and a launch waited
    assert max(gaps) < MOST
