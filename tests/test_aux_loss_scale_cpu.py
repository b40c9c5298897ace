"""The scale of the load-balancing loss may be a number or a tensor, which is not read on the host."""
import pytest
import torch

from primus_b200.models.moe import AuxLossScaler


@pytest.mark.parametrize("scale", [1, 0.25, torch.tensor(0.25), torch.tensor([0.5])])
def test_gradient_of_the_loss_is_the_scale(monkeypatch, scale):
    monkeypatch.setattr(AuxLossScaler, "scale", scale)
    x, aux = torch.ones(3, requires_grad=True), torch.zeros(1, requires_grad=True)
    AuxLossScaler.apply(x, aux).sum().backward()
    assert aux.grad.item() == float(scale) and (x.grad == 1).all()


def test_scale_on_a_device_is_not_read(monkeypatch):
    monkeypatch.setattr(AuxLossScaler, "scale", torch.ones((), device="meta"))      # (has no value to be read)
    x, aux = torch.ones(3, device="meta", requires_grad=True), torch.zeros(1, device="meta", requires_grad=True)
    AuxLossScaler.apply(x, aux).sum().backward()
    assert aux.grad.shape == (1,)
