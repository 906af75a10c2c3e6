"""Decays that underflow: sigmoid(log_lambda) of 0 has powers 0 (and 1 at a gate of exactly 0), in every engine,
and no gradient behind them is NaN."""

from __future__ import annotations

import contextlib

import pytest
import torch

from oracle import trunk_oracle as O
from tests.helpers import assert_close, build_trunk, norm_err, trunk_params

pytestmark = pytest.mark.gpu
DEV = "cuda"
B, N = 9, 5


def _trunk():
    trunk = build_trunk([128, 4, 1, 1, 1, 0])
    lru = trunk.yemong_layers[0].temporal[0].rg_lru
    with torch.no_grad():
        lru.log_lambda[:40] = torch.linspace(-120.0, -80.0, 40)   # 0 below -88.7, then denormal, then tiny
        lru.log_lambda[40] = 100.0
        lru.linear_a.bias[::3] = -200.0                           # recurrence gates of 0, some on dead decays
    return trunk


def _autocast(mode):
    return torch.autocast(DEV, dtype=torch.bfloat16) if mode == "bf16" else contextlib.nullcontext()


@pytest.mark.parametrize("mode", ["fp32", "bf16"])
@pytest.mark.parametrize("engine", ["auto", "simt"])
def test_step_with_dead_decays(mode, engine):
    from boost_and_broadside_b200 import _capi

    g = torch.Generator().manual_seed(1)
    x, hidden = torch.randn(B, N, 128, generator=g), torch.randn(1, B * N, 512, generator=g)
    alive = torch.ones(B, N, dtype=torch.bool)
    trunk = _trunk()
    ref = O.trunk_step(x, alive, hidden, trunk_params(trunk), 4, mode)
    assert all(torch.isfinite(t).all() for t in ref)
    trunk = trunk.to(DEV)
    with torch.no_grad(), _autocast(mode):
        got = trunk.step(x.to(DEV), alive.to(DEV), hidden.to(DEV), engine=_capi.ENGINE_SIMT if engine == "simt" else _capi.ENGINE_AUTO)
    for a, b, what in zip(got, ref, ("y", "hidden")):
        assert_close(a, b, mode, what)


@pytest.mark.parametrize("mode", ["fp32", "bf16"])
def test_training_with_dead_decays(mode):
    T = 4
    g = torch.Generator().manual_seed(2)
    x, hidden = torch.randn(T, B, N, 128, generator=g), torch.randn(1, B * N, 512, generator=g)
    alive = torch.ones(T, B, N, dtype=torch.bool)
    done = torch.rand(T, B, generator=g) < 0.2
    dy = torch.randn(T, B, N, 128, generator=g)
    trunk = _trunk()
    odx, odh, _, ograds = O.trunk_sequence_grad(x, alive, hidden, done, trunk_params(trunk), 4, dy, None)
    trunk = trunk.to(DEV).train()
    xg, hg = x.to(DEV).requires_grad_(), hidden.to(DEV).requires_grad_()
    with _autocast(mode):
        y, _ = trunk.sequence(xg, alive.to(DEV), hg, done.to(DEV))
    (y.float() * dy.to(DEV)).sum().backward()
    bound = 1e-4 if mode == "fp32" else 4e-2
    assert norm_err(xg.grad.cpu(), odx) <= bound and norm_err(hg.grad.cpu(), odh) <= bound
    for name, p in trunk.yemong_layers[0].named_parameters():
        if "field_sub" in name:
            continue
        ref = ograds[0][name]
        assert torch.isfinite(p.grad).all(), name
        told = torch.isfinite(ref)   # autograd of 0 ** c with respect to the 0 is inf * 0
        assert "log_lambda" in name or told.all()
        assert norm_err(p.grad.cpu()[told], ref[told]) <= bound, name


@pytest.mark.parametrize("mode", ["fp32", "bf16"])
def test_a_decay_that_is_not_a_number_stays_one(mode):
    trunk = _trunk()
    with torch.no_grad():
        trunk.yemong_layers[0].temporal[0].rg_lru.log_lambda[7] = float("nan")
    trunk = trunk.to(DEV)
    g = torch.Generator(device=DEV).manual_seed(3)
    with torch.no_grad(), _autocast(mode):
        _, h = trunk.step(torch.randn(B, N, 128, device=DEV, generator=g), None, torch.randn(1, B * N, 512, device=DEV, generator=g))
    assert torch.isnan(h[..., 7]).all() and torch.isfinite(h[..., 8:128]).all()
