"""The conv kernels of the differentiated sequence at row counts that give a thread more steps than it asks for at once (its loop goes
round, with a remainder), one and two segments, and blocks of the gradient a second turn over the rows, against the oracle's
autograd; episode boundaries around the steps where a turn begins."""

import pytest
import torch

from oracle import trunk_oracle as O
from tests.helpers import build_trunk, norm_err, trunk_params

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 2440 ship rows of 128 channels: 305 blocks of rows, above the chip's 296; 1200: 150, two segments; 32 channels: four times the rows for as many
@pytest.mark.parametrize("D,H,N,B,T", [(128, 4, 2, 1220, 5), (128, 4, 2, 1220, 9), (128, 4, 2, 1220, 13), (128, 4, 3, 400, 9), (128, 4, 3, 400, 13), (32, 4, 4, 2440, 13)])
def test_gradients_by_turns(D, H, N, B, T):
    gen = torch.Generator().manual_seed(D + B + T)
    trunk = build_trunk([D, H, 1, 1, 1, 0]).to(DEV).train()
    x = torch.randn(T, B, N, D, generator=gen)
    hidden = torch.randn(1, B * N, 4 * D, generator=gen) * 0.5
    alive = torch.ones(T, B, N, dtype=torch.bool)
    done = torch.rand(T, B, generator=gen) < 0.1
    done[3:5, 0::3] = True
    done[7:9, 1::3] = True
    dy, dh = torch.randn(x.shape, generator=gen), torch.randn(hidden.shape, generator=gen)
    params = trunk_params(trunk.cpu())
    trunk.to(DEV)
    odx, odh, _, ograds = O.trunk_sequence_grad(x, alive, hidden, done, params, H, dy, dh, None, None)
    xg, hg = x.to(DEV).requires_grad_(True), hidden.to(DEV).requires_grad_(True)
    y, h = trunk.sequence(xg, alive.to(DEV), hg, done.to(DEV))
    ((y * dy.to(DEV)).sum() + (h * dh.to(DEV)).sum()).backward()
    # the bound of the other oracle gradients; sums over up to 40 000 rows round to about 1e-6 of their size
    assert norm_err(xg.grad.cpu(), odx) < 1e-4
    assert norm_err(hg.grad.cpu(), odh) < 1e-4
    own, seen = dict(trunk.named_parameters()), 0
    for name, ref in ograds[0].items():
        if "conv" in name:
            seen += 1
            assert norm_err(own[f"yemong_layers.0.{name}"].grad.cpu(), ref) < 1e-4, name
    assert seen == 2
