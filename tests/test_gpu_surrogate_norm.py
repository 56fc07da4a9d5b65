"""Predictions under norms that the network's kernel does not take."""
import pytest
import torch

from psvwave_gb300 import surrogate

pytestmark = pytest.mark.gpu


def test_a_gradient_scale_being_fitted_stays_in_the_graph():
    net = surrogate.SurrogateNet(max_batch=8)
    z = torch.randn(5, 3, 20, 10, generator=torch.Generator().manual_seed(0)).cuda()
    scale = torch.linspace(0.5, 2.0, 600, device="cuda").reshape(3, 20, 10)
    net.norm["gs"] = scale.clone()
    m, g = net.predict(z)
    net.norm["gs"] = fitted = scale.clone().requires_grad_(True)
    m2, g2 = net.predict(z)
    assert torch.equal(m, m2) and torch.equal(g, g2.detach())
    g2.sum().backward()
    assert torch.allclose(fitted.grad * scale, g.sum(0), rtol=1e-5, atol=1e-6)
