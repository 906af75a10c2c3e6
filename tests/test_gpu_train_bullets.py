"""Bullets of the training path under bfloat16: rows of the slots in use only.  Counts around a block of keys (32) and a row tile
(128), no slot in use at all, every one, more than 16 tokens; both ways a differentiated call can run."""

import pytest
import torch

from tests.helpers import build_trunk, norm_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


def call(T, B, N, M, NB, mask, bullets, autocast):
    g = torch.Generator(device=DEV).manual_seed(T * 1000 + NB)
    trunk = build_trunk([128, 4, 2, 2, 1, 1]).to(DEV)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    x = r(T, B, N + M, 128).requires_grad_()
    hidden = 0.5 * r(2, B * N, 512)
    alive = torch.rand(T, B, N + M, device=DEV, generator=g) < 0.8
    alive[..., 0] = True
    bullets = bullets.clone().requires_grad_()
    dy = r(T, B, N + M, 128)
    with torch.autocast(DEV, dtype=torch.bfloat16, enabled=autocast):
        y, _ = trunk.sequence(x, alive, hidden, None, bullets=bullets, bullet_mask=mask)
    names = [n for n, _ in trunk.named_parameters() if M or "field_sub" not in n]
    params = dict(trunk.named_parameters())
    return dict(zip(["y", "x", "bullets", *names], [y.detach().float(), *torch.autograd.grad(y.float(), [x, bullets, *[params[n] for n in names]], dy, allow_unused=True)]))


@pytest.mark.parametrize("mode", ["keep", "recompute"])
@pytest.mark.parametrize("T,B,N,M,NB,density", [(1, 1, 1, 0, 1, 1.0), (2, 3, 12, 4, 31, 0.5), (2, 3, 12, 4, 33, 1.0), (1, 5, 8, 0, 70, 0.5), (2, 2, 17, 3, 80, 0.5),
                                                (3, 43, 3, 1, 20, 0.3), (1, 300, 2, 0, 9, 0.5), (2, 4, 8, 4, 16, 0.0)])
def test_masked_bullets(T, B, N, M, NB, density, mode, monkeypatch):
    monkeypatch.setenv("BNB_GRAD_MODE", mode)
    g = torch.Generator(device=DEV).manual_seed(NB)
    bullets = torch.randn(T * B, NB, 128, device=DEV, generator=g)
    mask = torch.rand(T * B, NB, device=DEV, generator=g) < density
    if density:
        mask[0] = True
        mask[-1] = T * B == 1
    half, full = call(T, B, N, M, NB, mask, bullets, True), call(T, B, N, M, NB, mask, bullets, False)
    assert not half["bullets"][~mask].any()
    for k, a in half.items():   # the bound of the other comparisons of the two precisions
        if a is not None and full[k] is not None and float(full[k].abs().max()) > 0:
            assert torch.isfinite(a).all(), k
            assert norm_err(a.float(), full[k].float()) < 4e-2, k
    # without a mask every slot is a key and no row moves: the same sums, the weights' in the order their atomics land
    every, none = call(T, B, N, M, NB, torch.ones_like(mask), bullets, True), call(T, B, N, M, NB, None, bullets, True)
    for k, a in every.items():
        if a is not None and float(none[k].abs().max()) > 0:
            assert norm_err(a.float(), none[k].float()) < 1e-4, k
