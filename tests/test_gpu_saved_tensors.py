"""What autograd promises around a differentiated trunk call: saved-tensor hooks see everything that is kept
for the backward, so that ``save_on_cpu`` and ``torch.utils.checkpoint`` free the device of it."""

from __future__ import annotations

import contextlib

import pytest
import torch

from tests.helpers import build_trunk

pytestmark = pytest.mark.gpu
DEV = "cuda"
T, B, N = 4, 33, 8


def _inputs(seed=0):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(T, B, N, 128, device=DEV, generator=gen)
    alive = torch.rand(T, B, N, device=DEV, generator=gen) < 0.9
    alive[..., 0] = True
    hidden = torch.randn(2, B * N, 512, device=DEV, generator=gen) * 0.5
    done = torch.rand(T, B, device=DEV, generator=gen) < 0.1
    dy = torch.randn(T, B, N, 128, device=DEV, generator=gen)
    return x.requires_grad_(True), alive, hidden, done, dy


def _autocast(bf16):
    return torch.autocast(DEV, dtype=torch.bfloat16) if bf16 else contextlib.nullcontext()


def _kept_bytes(bf16):
    from boost_and_broadside_b200 import _capi

    return _capi.lib.bnb_trunk_kept_bytes(2, 2, 1, 128, 4, _capi.uniform_batch(B, N, N), T, 0, _capi.BNB_BF16 if bf16 else _capi.BNB_FP32)


def _grads(trunk, run, seed=0):
    """Gradients of one call made by ``run``, and the bytes its forward left allocated."""
    x, alive, hidden, done, dy = _inputs(seed)
    params = [p for n, p in trunk.named_parameters() if "field_sub" not in n and "_bullet" not in n]
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    y, _ = run(x, alive, hidden, done)
    held = torch.cuda.memory_allocated() - before
    return [y.detach(), *torch.autograd.grad(y, [x, *params], dy)], held


def _assert_close(got, ref):
    for g, r in zip(got, ref):   # weight gradients are summed by atomics: their order is not fixed
        assert float((g - r).norm()) <= 1e-5 * float(r.norm()) + 1e-12


@pytest.fixture(autouse=True)
def _keep(monkeypatch):
    monkeypatch.setenv("BNB_GRAD_MODE", "keep")


@pytest.mark.parametrize("bf16", [False, True])
def test_saved_tensor_hooks_see_the_kept_activations(bf16):
    trunk = build_trunk([128, 4, 2, 2, 1, 0]).to(DEV)

    def plain(*a):
        with _autocast(bf16):
            return trunk.sequence(*a)

    ref, held = _grads(trunk, plain)
    assert held >= _kept_bytes(bf16)
    sizes = []

    def hooked(*a):
        # what is packed comes back somewhere else, off the boundary it was written on
        def pack(t):
            sizes.append(t.numel() * t.element_size())
            return t.cpu(), t

        def unpack(p):
            host, t = p
            if t.dtype != torch.uint8:
                return t
            return torch.empty(host.numel() + 16, dtype=torch.uint8, device=DEV)[16:].copy_(host)

        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            return plain(*a)

    got, _ = _grads(trunk, hooked)
    assert max(sizes) >= _kept_bytes(bf16)
    _assert_close(got, ref)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("how", ["save_on_cpu", "checkpoint"])
def test_kept_activations_leave_the_device_with_the_other_saved_tensors(bf16, how):
    from torch.utils.checkpoint import checkpoint

    trunk = build_trunk([128, 4, 2, 2, 1, 0]).to(DEV)

    def plain(*a):
        with _autocast(bf16):
            return trunk.sequence(*a)

    def moved(*a):
        if how == "checkpoint":   # the trunk is all of the region: its recomputation stops inside the call
            return checkpoint(plain, *a, use_reentrant=False)
        with torch.autograd.graph.save_on_cpu():
            return plain(*a)

    ref, _ = _grads(trunk, plain)
    got, held = _grads(trunk, moved)
    assert held < _kept_bytes(bf16) / 2
    _assert_close(got, ref)
    with pytest.raises(RuntimeError, match="another tensor"):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t.float() if t.dtype == torch.uint8 and t.dim() == 1 else t):
            _grads(trunk, plain)
