"""Sampling at counts around a warp, a block and more than the grid's
threads: sample i depends on the seed and i alone, so a shorter draw is the
start of a longer one; every outcome has weight, and on two amplitudes of
equal weight either comes up (exact comparisons throughout)."""
import pytest
import torch

from qcware_unitair_gb300.circuits import random_states
from qcware_unitair_gb300.measurement import sample

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("n", [8, 13, 18])
def test_shorter_draws_are_prefixes(n):
    psi = random_states(n, (), torch.complex64, seed=n).to(DEV)
    longest = sample(psi, 152 * 8 * 256 + 33, 7)
    assert int(longest.min()) >= 0 and int(longest.max()) < 2 ** n
    for count in (1, 31, 32, 33, 255, 257, 70001):
        assert torch.equal(sample(psi, count, 7), longest[:count])


def test_only_outcomes_with_weight():
    psi = torch.zeros(2 ** 14, dtype=torch.complex64, device=DEV)
    psi[3] = psi[16000] = 0.5 ** 0.5
    got = sample(psi, 5000, 1)
    assert sorted(set(got.tolist())) == [3, 16000]
