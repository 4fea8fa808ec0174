"""One circuit or program used on several streams: what is cached on it is
uploaded before another stream reads it.  Against the same calls one after another,
bit for bit (the same kernels on the same values)."""
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
