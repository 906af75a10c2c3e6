"""Bullet keys and values at the edges of their row tiles: active rows 0, 1, around one tile, above one tile per SM,
every row without a mask, both token types, environments around the single-CTA compaction, against the exact kernels."""

import pytest
import torch

from tests.helpers import build_trunk, norm_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,NB,active", [(3, 5, 0), (3, 5, 1), (2, 64, 127), (2, 64, 128), (3, 43, 129), (1, 1, None), (300, 80, 19000), (3, 43, None), (255, 3, 300), (256, 33, 3000), (257, 2, 200)])
def test_bullet_rows(B, NB, active, dtype):
    from boost_and_broadside_b200 import _capi

    g = torch.Generator(device=DEV).manual_seed(B + NB)
    trunk = build_trunk([128, 4, 1, 2, 1, 1]).to(DEV)
    x = torch.randn(B, 5, 128, device=DEV, generator=g)
    hidden = torch.randn(1, B * 4, 512, device=DEV, generator=g) * 0.5
    bullets = torch.randn(B, NB, 128, device=DEV, generator=g).to(dtype)
    mask = None
    if active is not None:
        mask = torch.zeros(B * NB, dtype=torch.bool, device=DEV)
        mask[torch.randperm(B * NB, device=DEV, generator=g)[:active]] = True
        mask = mask.view(B, NB)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        got = trunk.step(x, None, hidden, bullets=bullets, bullet_mask=mask)
        ref = trunk.step(x, None, hidden, engine=_capi.ENGINE_SIMT, bullets=bullets.float(), bullet_mask=mask)
    for a, b in zip(got, ref):
        assert norm_err(a.float(), b.float()) < 1e-2
