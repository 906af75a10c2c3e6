"""Callers that have to see the operators see them: function transforms, tracers and forward-mode
differentiation go through ``bnb_b200::*``, not past it into the native bodies."""

from __future__ import annotations

import pytest
import torch

from tests.helpers import build_trunk

pytestmark = pytest.mark.gpu
DEV = "cuda"
B, N = 6, 5


def _trunk_and_inputs(lead=()):
    trunk = build_trunk([128, 4, 2, 2, 1, 0]).to(DEV)
    gen = torch.Generator(device=DEV).manual_seed(3)
    x = torch.randn(*lead, B, N, 128, device=DEV, generator=gen)
    hidden = torch.randn(*lead, 2, B * N, 512, device=DEV, generator=gen)
    return trunk, x, hidden


def test_a_trace_holds_the_call_and_not_its_result():
    from torch.fx.experimental.proxy_tensor import make_fx

    trunk, x, hidden = _trunk_and_inputs()
    with torch.no_grad():
        step = lambda a, b: trunk.step(a, None, b)
        traced = make_fx(step)(x, hidden)
        assert any("trunk_forward" in str(n.target) for n in traced.graph.nodes)
        x2, h2 = x.flip(0).contiguous(), hidden * 0.5
        for got, ref in zip(traced(x2, h2), step(x2, h2)):
            assert torch.equal(got, ref)


def test_transforms_that_the_operators_do_not_take_raise():
    trunk, x, hidden = _trunk_and_inputs((3,))
    step = lambda a, b: trunk.step(a, None, b)
    with torch.no_grad():
        with pytest.raises(RuntimeError):   # no batching rule for an operator with lists
            torch.vmap(step)(x, hidden)
        with pytest.raises(RuntimeError):   # TorchScript has no node for it
            torch.jit.trace(step, (x[0], hidden[0]), check_trace=False)
        step(x[0], hidden[0])               # and nothing is left behind


@pytest.mark.parametrize("mode", ["keep", "recompute"])
def test_forward_mode_derivatives_are_refused(mode, monkeypatch):
    monkeypatch.setenv("BNB_GRAD_MODE", mode)
    import torch.autograd.forward_ad as fwad

    trunk, x, hidden = _trunk_and_inputs()
    with fwad.dual_level():
        dual = fwad.make_dual(x, torch.ones_like(x))
        with pytest.raises((NotImplementedError, RuntimeError), match="jvp|forward"):
            trunk.sequence(dual[None], None, hidden, None)


def test_heads_under_vmap():
    import boost_and_broadside_b200 as bnb

    head = bnb.HeadMLP(128, 12).to(DEV)
    x = torch.randn(3, 7, 128, device=DEV)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        y = torch.vmap(head)(x)
        for i in range(3):
            assert torch.equal(y[i], head(x[i]))
