"""The native host path against the Python functions it stands in for, bit
for bit, over the forms both accept: dtypes, batch forms, strides, offsets,
kinds of qubit sequence, parameters, subclasses, modes and transforms, with
and without gradients."""
import contextlib

import numpy as np
import pytest
import torch

import qcware_unitair_gb300 as ug
from qcware_unitair_gb300 import _native

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@contextlib.contextmanager
def python_path(monkeypatch):
    with monkeypatch.context() as m:
        for name in _native.NAMES:
            m.setattr(_native, name, lambda *a: None)
        yield


def rand(rng, shape, dtype):
    a = rng.normal(size=shape)
    if dtype.is_complex:
        a = a + 1j * rng.normal(size=shape)
    return torch.from_numpy(np.asarray(a)).to(dtype).to(DEV)


def strided(t):
    """The same values in a tensor that is not contiguous."""
    buf = torch.zeros(t.shape + (2,), dtype=t.dtype, device=t.device)
    buf[..., 0] = t
    return buf[..., 0]


def offset(t):
    buf = torch.zeros(t.numel() + 1, dtype=t.dtype, device=t.device)
    buf[1:] = t.reshape(-1)
    return buf[1:].view(t.shape)


def both(monkeypatch, call, inputs, grad):
    """Outputs and input gradients of the native and the Python path."""
    got = []
    for native in (True, False):
        ctx = contextlib.nullcontext() if native else python_path(monkeypatch)
        with ctx:
            xs = [t.detach().requires_grad_(grad and t.dtype.is_floating_point
                                            or grad and t.dtype.is_complex)
                  for t in inputs]
            try:
                out = call(*xs)
                if grad:
                    w = torch.linspace(0.5, 1.5, out.numel(), device=DEV,
                                       dtype=torch.float64).view(out.shape)
                    out.backward(w.to(out.dtype))
            except RuntimeError as e:  # refused: by both alike
                got.append((type(e), str(e)))
                continue
            got.append([out.detach()] + [x.grad for x in xs])
    if isinstance(got[0], tuple) or isinstance(got[1], tuple):
        assert got[0] == got[1]
        return None
    for a, b in zip(*got):
        assert (a is None) == (b is None)
        if a is not None:
            assert a.shape == b.shape and a.dtype == b.dtype
            assert torch.equal(a, b)
    return got[0][0]


SHAPES = [((), ()), ((3,), (3,)), ((), (3,)), ((3,), ()), ((2, 3), (2, 3)),
          ((1,), (3,)), ((3,), (2, 3)), ((1, 3), (3,)), ((1,), (1,)),
          ((1,), ())]


@pytest.mark.parametrize("ob,sb", SHAPES)
@pytest.mark.parametrize("k", [0, 1, 2, 3, 5, 6])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("form", [lambda t: t, strided, offset])
def test_apply_operator(monkeypatch, ob, sb, k, dtype, grad, form):
    n = 7
    rng = np.random.default_rng(k)
    m = form(rand(rng, ob + (2 ** k, 2 ** k), dtype))
    s = form(rand(rng, sb + (2 ** n,), dtype))
    qs = [int(q) for q in rng.choice(n, size=k, replace=False)]
    for q in (qs, tuple(qs), np.array(qs, dtype=np.int64), iter(qs)) \
            if not grad else (qs,):
        q = list(q) if not isinstance(q, (list, tuple, np.ndarray)) else q
        both(monkeypatch, lambda a, b: ug.apply_operator(a, q, b), (m, s),
             grad)


@pytest.mark.parametrize("ob,sb", SHAPES)
@pytest.mark.parametrize("n", [1, 3, 9, 13])
@pytest.mark.parametrize("each", [False, True])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("grad", [False, True])
def test_layers(monkeypatch, ob, sb, n, each, dtype, grad):
    rng = np.random.default_rng(n)
    m = rand(rng, ob + ((n,) if each else ()) + (2, 2), dtype)
    s = rand(rng, sb + (2 ** n,), dtype)
    fn = ug.apply_each_qubit if each else ug.apply_all_qubits
    both(monkeypatch, fn, (m, s), grad)


@pytest.mark.parametrize("sa,ss", [((), (8,)), ((8,), (8,)), ((8,), (3, 8)),
                                   ((3, 1), (3, 8)), ((5, 8), (8,)),
                                   ((2, 1, 8), (3, 8)), ((1,), (8,)),
                                   ((3, 8), (3, 1))])
@pytest.mark.parametrize("da", [torch.float32, torch.float64, torch.float16,
                                torch.int64])
@pytest.mark.parametrize("ds", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("form", [lambda t: t, strided])
def test_apply_phase(monkeypatch, sa, ss, da, ds, grad, form):
    rng = np.random.default_rng(1)
    a = form((rand(rng, sa, torch.float64) * 3).to(da))
    both(monkeypatch, ug.apply_phase, (a, form(rand(rng, ss, ds))), grad)


@pytest.mark.parametrize("sa,ss", [((8,), (8,)), ((8,), (3, 8)),
                                   ((3, 1), (3, 8)), ((5, 8), (8,)),
                                   ((2, 1, 8), (3, 8)), ((1,), (8,)),
                                   ((20000,), (2, 20000)), ((1,), (1,))])
@pytest.mark.parametrize("ds", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("dd", [torch.float32, torch.float64])
@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("form", [lambda t: t, strided])
def test_reductions(monkeypatch, sa, ss, ds, dd, grad, form):
    rng = np.random.default_rng(2)
    s = form(rand(rng, ss, ds))
    both(monkeypatch, ug.diag_expectation_value, (rand(rng, sa, dd), s), grad)
    both(monkeypatch, ug.inner_product, (form(rand(rng, sa, ds)), s), grad)
    both(monkeypatch, ug.norm_squared, (s,), grad)
    both(monkeypatch, ug.abs_squared, (s,), grad)


def test_refusals_are_the_same(monkeypatch):
    c64, c128 = torch.complex64, torch.complex128
    m = torch.eye(2, dtype=c64, device=DEV)
    s = torch.ones(8, dtype=c64, device=DEV)
    calls = [
        lambda: ug.apply_operator(m, [3], s),
        lambda: ug.apply_operator(m, [-1], s),
        lambda: ug.apply_operator(m, [0, 1], s),
        lambda: ug.apply_operator(torch.eye(4, dtype=c64, device=DEV),
                                  [1, 1], s),
        lambda: ug.apply_operator(m.to(c128), [0], s),
        lambda: ug.apply_operator(m, [0], s[:5]),
        lambda: ug.apply_operator(m[:, :1], [0], s),
        lambda: ug.apply_operator(m.cpu(), [0], s),
        lambda: ug.apply_operator(m.real, [0], s.real),
        lambda: ug.apply_operator(m.expand(3, 2, 2), [0], s.expand(2, 8)),
        lambda: ug.apply_operator(m[0], [0], s),
        lambda: ug.apply_all_qubits(torch.eye(4, dtype=c64, device=DEV), s),
        lambda: ug.apply_all_qubits(m, s[:1]),
        lambda: ug.apply_each_qubit(m.expand(2, 2, 2), s),
        lambda: ug.apply_phase(s, s),
        lambda: ug.apply_phase(torch.ones(3, device=DEV), s),
        lambda: ug.inner_product(s, s.to(c128)),
        lambda: ug.inner_product(s, s[:3]),
        lambda: ug.diag_expectation_value(s, s),
        lambda: ug.norm_squared(s.real)]
    for i, call in enumerate(calls):
        errors = []
        for native in (True, False):
            ctx = contextlib.nullcontext() if native else \
                python_path(monkeypatch)
            with ctx, pytest.raises(Exception) as e:
                call()
            errors.append((e.type, str(e.value)))
        assert errors[0] == errors[1], i


def test_what_is_left_to_python():
    """Parameters take the native path; subclasses, lazily conjugated
    tensors, modes, transforms and tracers do not."""
    mod = _native.load()
    m = torch.eye(2, dtype=torch.complex64, device=DEV)
    s = torch.ones(8, dtype=torch.complex64, device=DEV)
    assert mod.apply_operator(torch.nn.Parameter(m), [0], s) is not None
    with torch.inference_mode():
        assert mod.apply_operator(m, range(1), s.clone()) is not None

    class Sub(torch.Tensor):
        pass

    assert mod.apply_operator(m.as_subclass(Sub), [0], s) is None
    assert mod.apply_operator(m.conj(), [0], s) is None
    assert mod.apply_operator(m, iter([0]), s) is None
    assert mod.apply_operator(m, [np.int64(0)], s) is None
    assert mod.apply_operator(m, [True], s) is None
    from torch.utils._python_dispatch import TorchDispatchMode

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Mode():
        assert mod.apply_operator(m, [0], s) is None
    seen = []

    def f(x):
        seen.append(mod.norm_squared(x))
        return x

    torch.vmap(f)(s.view(2, 4))
    assert seen == [None]
    import torch.autograd.forward_ad as fwd
    with fwd.dual_level():
        assert mod.norm_squared(fwd.make_dual(s, s)) is None


def test_create_graph_and_saved_tensor_hooks(monkeypatch):
    s = torch.randn(3, 16, dtype=torch.complex128, device=DEV)
    d = torch.randn(16, dtype=torch.float64, device=DEV)
    got = []
    for native in (True, False):
        ctx = contextlib.nullcontext() if native else python_path(monkeypatch)
        with ctx:
            x = s.clone().requires_grad_()
            packed = []
            with torch.autograd.graph.saved_tensors_hooks(
                    lambda t: packed.append(t.shape) or t, lambda t: t):
                e = ug.diag_expectation_value(d, x) * ug.norm_squared(x) + \
                    ug.abs_squared(x).sum(-1) + ug.inner_product(x, x).real
            g, = torch.autograd.grad(e.sum(), x, create_graph=True)
            h, = torch.autograd.grad(g.abs().square().sum(), x)
            got.append((g.detach(), h, sorted(packed)))
    assert torch.equal(got[0][0], got[1][0])
    assert torch.equal(got[0][1], got[1][1])
    assert got[0][2] == got[1][2]


def test_streams_and_threads():
    """Calls from several threads on their own streams, with gradients."""
    import threading
    m = torch.linalg.qr(torch.randn(4, 4, dtype=torch.complex64,
                                    device=DEV))[0]
    s = torch.randn(5, 2 ** 12, dtype=torch.complex64, device=DEV)
    torch.cuda.synchronize()

    def work(out, i):
        st = torch.cuda.Stream(DEV)
        with torch.cuda.stream(st):
            x = s.clone().requires_grad_()
            op = m.clone().requires_grad_()
            y = x
            for q in range(10):
                y = ug.apply_operator(op, [q, q + 1], y)
            ug.norm_squared(y[:, :100].contiguous().view(5, 100)).sum() \
                .backward()
            st.synchronize()
            out[i] = (x.grad, op.grad)

    out = {}
    ts = [threading.Thread(target=work, args=(out, i)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for i in range(1, 4):
        assert torch.equal(out[i][0], out[0][0])
        assert torch.equal(out[i][1], out[0][1])
