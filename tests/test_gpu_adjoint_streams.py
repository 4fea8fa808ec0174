"""One circuit evaluated on several streams and threads at once: each call's
rotation values are its own, and what is cached on the circuit is uploaded
before another stream reads it.  Against the same calls one after another,
bit for bit (the same kernels on the same values)."""
import threading

import pytest
import torch

from qcware_unitair_gb300 import adjoint as ad
from qcware_unitair_gb300.fusion import Circuit

pytestmark = pytest.mark.gpu
DEV = "cuda"
CALLS = 6


def circuit(n, layers):
    pc = ad.hardware_efficient_ansatz(n, layers)
    pc.rx(0, 0)
    return pc, ad.PauliSum(n).z(0).xx(0, n - 1, 0.5)


def inputs(pc, batch):
    g = torch.Generator().manual_seed(3)
    return [torch.randn(batch, pc.num_params, generator=g,
                        dtype=torch.float64).to(DEV) for _ in range(CALLS)]


def evaluate(pc, H, params):
    p = params.clone().requires_grad_()
    value = ad.expectation(pc, p, H)
    value.sum().backward()
    return value.detach(), p.grad


def busy(ms):
    """Work that keeps the stream behind for a while."""
    x = torch.randn(2048, 2048, device=DEV)
    for _ in range(int(4 * ms)):
        x = (x @ x).clamp(-1, 1)


def same(got, want):
    for g, w in zip(got, want):
        for a, b in zip(g, w):
            assert torch.equal(a, b)


@pytest.mark.parametrize("n,layers,batch", [(6, 3, 4), (14, 4, 8)])
def test_streams(n, layers, batch):
    pc, H = circuit(n, layers)
    params = inputs(pc, batch)
    want = [evaluate(pc, H, p) for p in params]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(CALLS)]
    for _ in range(3):
        got = []
        for s, p in zip(streams, params):
            with torch.cuda.stream(s):
                got.append(evaluate(pc, H, p))
        torch.cuda.synchronize()
        same(got, want)


@pytest.mark.parametrize("n,layers,batch", [(6, 3, 4), (12, 4, 8)])
def test_threads_on_one_stream(n, layers, batch):
    pc, H = circuit(n, layers)
    params = inputs(pc, batch)
    want = [evaluate(pc, H, p) for p in params]
    torch.cuda.synchronize()
    for _ in range(3):
        got = [None] * CALLS
        start = threading.Barrier(CALLS)

        def run(i):
            start.wait()
            got[i] = evaluate(pc, H, params[i])

        threads = [threading.Thread(target=run, args=(i,))
                   for i in range(CALLS)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        same(got, want)


@pytest.mark.parametrize("first", [0, 1])
def test_cached_uploads_behind_other_work(first):
    """The first call, on a stream that is behind, plans and uploads; the
    second, on an idle stream, must not read before the copies."""
    pc, H = circuit(13, 4)
    params = inputs(pc, 4)
    want = evaluate(*circuit(13, 4), params[1])
    torch.cuda.synchronize()
    late, idle = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(late):
        busy(30)
        if first:
            evaluate(pc, H, params[0])
        else:
            ad.expectation(pc, params[0], H)
    with torch.cuda.stream(idle):
        got = evaluate(pc, H, params[1])
    torch.cuda.synchronize()
    same([got], [want])


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("fuse", [True, False])
def test_program_on_another_stream(fuse, dtype):
    n = 13
    c = Circuit(n)
    for q in range(n):
        c.h(q).rz(q, 0.1 * q).cnot(q, (q + 1) % n)
    x = torch.zeros(2 ** n, dtype=dtype, device=DEV)
    x[0] = 1
    want = c.compile(dtype, DEV, fuse=fuse).run(x)
    torch.cuda.synchronize()
    late, idle = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(late):
        busy(30)
        prog = c.compile(dtype, DEV, fuse=fuse)
    with torch.cuda.stream(idle):
        got = prog.run(x)
        del prog
    torch.cuda.synchronize()
    assert torch.equal(got, want)


def test_capture_after_another_stream():
    """A circuit that was run on one stream, captured on another."""
    pc, H = circuit(10, 3)
    params = inputs(pc, 4)
    want = [ad.expectation(pc, p, H) for p in params]
    torch.cuda.synchronize()
    p = params[0].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = ad.expectation(pc, p, H)
    for new, w in zip(params, want):
        p.copy_(new)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, w)
