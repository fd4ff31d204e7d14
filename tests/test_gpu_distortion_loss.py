"""What the fused distortion loss has to share with the torch expression it stands for beyond its value at finite inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _expression(d):
    total = (d[:, :, 2] ** 2).clip(min=1e-6)
    return (((d[:, :, 0] - d[:, :, 1]) + d[:, :, 4]) / total).clip(min=0).mean()


@pytest.mark.parametrize("channel", range(5))
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
def test_non_finite_moments(cuda_lib, channel, value):
    """A diverged pixel shows in the loss and in its gradient wherever it does in torch."""
    from radiance_meshes_b200.render import DistortionLoss
    d = torch.rand((9, 33, 5), generator=torch.Generator().manual_seed(channel)).to("cuda:0") + 0.1
    d[4, 5, channel] = value
    out = []
    for loss in (DistortionLoss.apply, _expression):
        x = d.clone().requires_grad_(True)
        y = loss(x)
        y.backward()
        out.append((y.detach(), x.grad))
    for got, want in zip(*out):
        # float32 on both sides: the sum over the pixels in another order, a gradient's products in another
        assert torch.allclose(got, want, rtol=1e-5, atol=0.0, equal_nan=True), (got[4, 5], want[4, 5]) if got.dim() else (got, want)


def test_gradient_can_be_differentiated_again(cuda_lib):
    """A penalty on the loss's gradient (create_graph), through the moments and through the factor of the loss."""
    from radiance_meshes_b200.render import DistortionLoss
    d = torch.rand((7, 21, 5), generator=torch.Generator().manual_seed(3)).to("cuda:0") + 0.1
    out = []
    for loss in (DistortionLoss.apply, _expression):
        x, k = d.clone().requires_grad_(True), torch.tensor(3.0, device="cuda:0", requires_grad=True)
        first, = torch.autograd.grad(k * loss(2.0 * x), x, create_graph=True)
        (first ** 2).sum().backward()
        out.append((first.detach(), x.grad, k.grad))
    for got, want in zip(*out):
        assert torch.allclose(got, want, rtol=1e-4, atol=0.0)  # float32: two quotients and their sums
