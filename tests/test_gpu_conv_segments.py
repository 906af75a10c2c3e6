"""The conv kernels of the differentiated sequence where a thread's segment of steps begins and ends: 1 to 3 steps (the state's
taps come back among its own), one, two and uneven segments, boundaries in every step around them, against the oracle's
autograd; widths whose rows are not a power of two of quads."""

import pytest
import torch

from oracle import trunk_oracle as O
from tests.helpers import build_trunk, norm_err, trunk_params

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dims", [[128, 4, 1, 1, 1, 0, 3, 0], [96, 3, 1, 1, 1, 0, 2, 1], [32, 4, 1, 1, 1, 0, 5, 0]])
@pytest.mark.parametrize("T", [1, 2, 3, 4, 5, 8, 9, 12, 13, 33])
def test_sequence_gradients_by_steps(dims, T):
    D, H, N, M, B = dims[0], dims[1], dims[6], dims[7], 4
    gen = torch.Generator().manual_seed(D + T)
    trunk = build_trunk(dims).to(DEV).train()
    x = torch.randn(T, B, N + M, D, generator=gen)
    hidden = torch.randn(1, B * N, 4 * D, generator=gen) * 0.5
    alive = torch.ones(T, B, N + M, dtype=torch.bool)
    done = torch.rand(T, B, generator=gen) < 0.3
    done[:, 0], done[:, 1] = False, True
    dy, dh = torch.randn(x.shape, generator=gen), torch.randn(hidden.shape, generator=gen)
    params = trunk_params(trunk.cpu())
    trunk.to(DEV)
    odx, odh, _, ograds = O.trunk_sequence_grad(x, alive, hidden, done, params, H, dy, dh, None, None)
    xg, hg = x.to(DEV).requires_grad_(True), hidden.to(DEV).requires_grad_(True)
    y, h = trunk.sequence(xg, alive.to(DEV), hg, done.to(DEV))
    ((y * dy.to(DEV)).sum() + (h * dh.to(DEV)).sum()).backward()
    # float32 products and sums of a few dozen rows: the bound of the other gradient tests
    assert norm_err(xg.grad.cpu(), odx) < 1e-4
    assert norm_err(hg.grad.cpu(), odh) < 1e-4
    own = dict(trunk.named_parameters())
    seen = 0
    for block, grads in enumerate(ograds):
        for name, ref in grads.items():
            if "conv" in name:
                seen += 1
                assert norm_err(own[f"yemong_layers.{block}.{name}"].grad.cpu(), ref) < 1e-4, name
    assert seen == 2
