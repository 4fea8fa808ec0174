"""The adjoint calls' parameters: too few are refused on the host (the
kernels would read past the rows), more than the circuit has are left out of
its values and its gradients."""
import pytest
import torch

from qcware_unitair_gb300 import adjoint as ad


class Cuda(torch.Tensor):
    """A host tensor that says it is on the device: the check comes before
    any launch."""
    is_cuda = True


@pytest.mark.parametrize("shape", [(2, 5), (6,), (2, 1, 6), (2, 0)])
def test_too_few_parameters(shape):
    pc = ad.ParamCircuit(3, 6)
    pc.rx(0, 5)
    for fn in (ad.expectation_and_grad, ad.evaluate, ad.expectation):
        with pytest.raises(ValueError, match="params must be"):
            fn(pc, torch.zeros(shape).as_subclass(Cuda), ad.PauliSum(3).z(0))


@pytest.mark.gpu
@pytest.mark.parametrize("fuse", [True, False])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_more_parameters(dtype, fuse):
    n, batch = 10, 3
    pc = ad.hardware_efficient_ansatz(n, 2)
    g = torch.Generator().manual_seed(1)
    wide = torch.randn(batch, pc.num_params + 7, generator=g).to(dtype).cuda()
    H = ad.PauliSum(n).z(0).xx(0, 1, 0.5)
    want = ad.expectation_and_grad(pc, wide[:, :pc.num_params].contiguous(),
                                   H, fuse=fuse)
    got = ad.expectation_and_grad(pc, wide, H, fuse=fuse)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    assert torch.equal(ad.evaluate(pc, wide, H),
                       ad.evaluate(pc, wide[:, :pc.num_params], H))
