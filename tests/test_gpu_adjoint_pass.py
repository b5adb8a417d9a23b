"""The autograd function's gradient does not depend on what happened to the
library's one kept pass between forward and backward: kept, replaced by another
forward call, consumed by an earlier backward call, or its object made anew."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from tealeaf_opencl_gb300 import adjoint, lib  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(7, 33), (130, 257)])
def test_gradient_with_the_pass_kept_replaced_and_consumed(shape):
    g = torch.Generator(device="cuda").manual_seed(3)
    theta, energy, obs = (torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)
                          for _ in range(3))
    energy, obs = energy.exp(), obs.exp()
    lib.load().tea_gb300_set_arithmetic(1)
    adj = lib.Adjoint(shape[1], shape[0])
    cfg = adj.config(5, 0.004, 1e-12, 5000, 2)

    def forward(t):
        t = t.detach().requires_grad_(True)
        return t, adjoint.time_stepped_loss(t, energy, obs, adj, cfg)

    try:
        t, loss = forward(theta)
        loss.backward(retain_graph=True)
        want = t.grad.clone()
        t.grad = None
        loss.backward()  # the pass was consumed
        assert torch.equal(t.grad, want)
        t, loss = forward(theta)
        forward(theta + 1.0)  # replaced
        loss.backward()
        assert torch.equal(t.grad, want)
        t, loss = forward(theta)
        adj = lib.Adjoint(shape[1], shape[0])  # the library's object made anew
        loss.backward()
        assert torch.equal(t.grad, want)
        assert np.isfinite(want.cpu().numpy()).all() and float(want.abs().max()) > 0.0
    finally:
        adj.free()
