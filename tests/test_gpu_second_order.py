"""A second-order gradient through the trunk is refused, not dropped; a first-order one with create_graph is
not."""

from __future__ import annotations

import pytest
import torch

from tests.helpers import build_trunk

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("mode", ["keep", "recompute"])
@pytest.mark.parametrize("through", ["x", "parameter", "incoming"])
def test_second_order_gradients_raise(mode, through, monkeypatch):
    monkeypatch.setenv("BNB_GRAD_MODE", mode)
    T, B, N = 2, 5, 4
    trunk = build_trunk([128, 4, 2, 2, 1, 0]).to(DEV)
    gen = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(T, B, N, 128, device=DEV, generator=gen, requires_grad=True)
    hidden = torch.randn(2, B * N, 512, device=DEV, generator=gen)
    dy = torch.randn(T, B, N, 128, device=DEV, generator=gen, requires_grad=True)
    p = trunk.yemong_layers[1].spatial[1].out_proj.weight

    def first(create_graph):
        y, _ = trunk.sequence(x, None, hidden, None)
        return y, torch.autograd.grad(y, [x, p], dy, create_graph=create_graph, retain_graph=True)

    _, plain = first(False)
    assert not any(g.requires_grad for g in plain)
    y, recorded = first(True)
    assert all(g.requires_grad for g in recorded)
    for a, b in zip(recorded, plain):
        assert float((a - b).detach().norm()) <= 1e-5 * float(b.norm())
    # the penalty alone: y's own backward would find its activations consumed
    penalty = recorded[0].square().sum() + recorded[1].square().sum()
    with pytest.raises(RuntimeError, match="differentiated again|no autograd formula"):
        torch.autograd.grad(penalty, {"x": x, "parameter": p, "incoming": dy}[through])
