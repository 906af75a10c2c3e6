"""Training attention over bullets against the oracle's autograd where the keys of an environment-step fill one block of 32, more than one
and several, so that the running softmax is rescaled and the gradient takes its two sweeps: up to 8, 16 and 32 tokens, an
environment-step without a bullet, one with all of them."""

import pytest
import torch

from oracle import trunk_oracle as O
from tests.helpers import build_trunk, norm_err, trunk_params

pytestmark = pytest.mark.gpu
DEV = "cuda"


# float32: sums of a few hundred terms, the bound of the other oracle gradients; bfloat16: the bound of the comparisons of the two precisions
@pytest.mark.parametrize("route,bound", [("float32", 1e-4), ("keep", 4e-2), ("recompute", 4e-2)])
@pytest.mark.parametrize("N,M,NB", [(4, 0, 33), (7, 1, 64), (8, 0, 110), (9, 0, 65), (12, 4, 33), (13, 2, 110), (20, 3, 65)])
def test_gradients_by_active_keys(N, M, NB, route, bound, monkeypatch):
    if route != "float32":
        monkeypatch.setenv("BNB_GRAD_MODE", route)
    T, B = 2, 3
    gen = torch.Generator().manual_seed(100 * N + NB)
    trunk = build_trunk([128, 4, 1, 2, 1, 1]).to(DEV).train()
    x = torch.randn(T, B, N + M, 128, generator=gen)
    alive = torch.rand(T, B, N + M, generator=gen) < 0.8
    alive[..., 0] = True
    hidden = torch.randn(1, B * N, 512, generator=gen) * 0.5
    bullets = torch.randn(T * B, NB, 128, generator=gen)
    mask = torch.rand(T * B, NB, generator=gen) < 0.7
    mask[0], mask[1] = False, True
    dy, dh = torch.randn(x.shape, generator=gen), torch.randn(hidden.shape, generator=gen)
    params = trunk_params(trunk.cpu())
    trunk.to(DEV)
    odx, odh, odb, ograds = O.trunk_sequence_grad(x, alive, hidden, None, params, 4, dy, dh, bullets, mask)
    xg, hg, bg = (t.to(DEV).requires_grad_(True) for t in (x, hidden, bullets))
    with torch.autocast(DEV, dtype=torch.bfloat16, enabled=route != "float32"):
        y, h = trunk.sequence(xg, alive.to(DEV), hg, None, bullets=bg, bullet_mask=mask.to(DEV))
    ((y * dy.to(DEV)).sum() + (h * dh.to(DEV)).sum()).backward()
    assert not bg.grad[~mask.to(DEV)].any()
    for name, got, ref in (("x", xg, odx), ("hidden", hg, odh), ("bullets", bg, odb)):
        assert norm_err(got.grad.cpu(), ref) < bound, name
    own, seen = dict(trunk.named_parameters()), 0
    for name, ref in ograds[0].items():
        if name.startswith("spatial.0.") and float(ref.abs().max()) > 0:
            seen += 1
            assert norm_err(own[f"yemong_layers.0.{name}"].grad.cpu(), ref) < bound, name
    assert seen >= 8
