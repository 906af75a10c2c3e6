"""The attention kernel beside the tile kernel at the edges of its blocks of keys (32, the last up to 16 by themselves) and of its
stages of 48 bullets, against the oracle; an environment without a live ship, one without bullets, one with all of them."""

import pytest
import torch

from oracle import trunk_oracle as O
from tests.helpers import assert_close, build_trunk, trunk_params

pytestmark = pytest.mark.gpu
DEV = "cuda"


# tokens: one pair of head and query block a warp up to 16, several above; above 128 without bullets too
@pytest.mark.parametrize("tokens,slots", [(1, 1), (5, 16), (12, 17), (15, 32), (16, 33), (16, 48), (12, 49), (8, 96), (12, 97), (3, 160), (17, 49),
                                          (32, 64), (33, 100), (48, 15), (65, 47), (129, 0), (144, 0), (145, 0), (177, 0)])
@pytest.mark.parametrize("masked", [True, False])
def test_step_by_keys_and_bullets(tokens, slots, masked):
    if not slots and not masked:
        pytest.skip("no bullets to mask")
    gen = torch.Generator().manual_seed(1000 * tokens + slots)
    envs = 5
    trunk = build_trunk([128, 4, 1, 2, 1, 1])
    params = trunk_params(trunk)
    x = torch.randn(envs, tokens, 128, generator=gen)
    alive = torch.rand(envs, tokens, generator=gen) < 0.7
    alive[0] = False
    hidden = torch.randn(1, envs * tokens, 512, generator=gen) * 0.5
    bullets = torch.randn(envs, slots, 128, generator=gen) if slots else None
    mask = None
    if slots and masked:
        mask = torch.rand(envs, slots, generator=gen) < 0.5
        mask[1] = False
        mask[2] = True
    ref_y, ref_h = O.trunk_step(x, alive, hidden, params, 4, "bf16", bullets, mask)
    trunk = trunk.to(DEV)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        y, h = trunk.step(x.to(DEV), alive.to(DEV), hidden.to(DEV), bullets=None if bullets is None else bullets.to(DEV),
                          bullet_mask=None if mask is None else mask.to(DEV))
    assert_close(y, ref_y, "bf16", "y")
    assert_close(h, ref_h, "bf16", "hidden")
