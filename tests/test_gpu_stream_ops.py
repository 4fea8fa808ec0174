"""3- to 5-qubit complex64 operators in warp steps (dense_stream_kernel)
against the kernels that take unaligned states: equal bit for bit (each output
sums the same products in the same order), from the smallest state it takes
(one step) over several steps per warp, targets on the lowest, highest and
mixed bits in any order, batches, broadcast states and in place."""
import numpy as np
import pytest
import torch

import qcware_unitair_gb300 as ug

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _rand(rng, *shape):
    return torch.from_numpy(rng.normal(size=shape) + 1j * rng.normal(
        size=shape)).to(torch.complex64).to(DEV)


def _unaligned(t):
    buf = torch.zeros(t.numel() + 1, dtype=t.dtype, device=t.device)
    buf[1:] = t.reshape(-1)
    return buf[1:].view(t.shape)


@pytest.mark.parametrize("k", [3, 4, 5])
@pytest.mark.parametrize("extra", [5, 6, 9, 14])
@pytest.mark.parametrize("batch", [(), (1,), (3,)])
@pytest.mark.parametrize("where", ["low", "high", "ends", "random", "other"])
def test_matches_the_unaligned_kernels(k, extra, batch, where):
    n = k + extra
    rng = np.random.default_rng(n)
    qs = {"low": list(range(n - k, n)), "high": list(range(k))[::-1],
          "ends": ([0, n - 1, 1, n - 2, 2])[:k],
          "random": [int(q) for q in rng.choice(n, k, replace=False)],
          "other": [int(q) for q in rng.permutation(n)[:k]]}[where]
    m, s = _rand(rng, 2 ** k, 2 ** k), _rand(rng, *batch, 2 ** n)
    got = ug.apply_operator(m, qs, s)
    ref = ug.apply_operator(m, qs, _unaligned(s))
    assert torch.equal(got, ref)
    inplace = s.clone()
    ug.apply_operator_(m, qs, inplace)
    assert torch.equal(inplace, ref)


@pytest.mark.parametrize("k", [3, 4, 5])
def test_broadcast_state_and_many_steps(k):
    rng = np.random.default_rng(k)
    n = 20
    m = _rand(rng, 2 ** k, 2 ** k)
    s = _rand(rng, 5, 2 ** n)
    qs = [int(q) for q in rng.choice(n, k, replace=False)]
    ref = torch.stack([ug.apply_operator(m, qs, _unaligned(x)) for x in s])
    assert torch.equal(ug.apply_operator(m, qs, s), ref)
    # one state under a batch of operators keeps the per-state kernels
    ops = m.expand(3, -1, -1).contiguous()
    got = ug.apply_operator(ops, qs, s[0])
    assert (got - ref[0]).abs().max() <= 2e-6 * ref.abs().max() * 2 ** (k / 2)
