"""Attention inside a tile: environments that share a block of 16 queries (up to 8 tokens), that fill one, and that walk
several, at every size where the number per block or per tile changes, with a last tile that is not full and an
environment without a live key."""

import pytest
import torch

from oracle import trunk_oracle as O
from tests.helpers import assert_close, build_trunk, trunk_params

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("tokens", [1, 2, 3, 5, 7, 8, 9, 15, 16, 17, 33, 64, 65, 128])
def test_step_against_the_oracle_by_environment_size(tokens):
    gen = torch.Generator().manual_seed(tokens)
    envs = 2 * (128 // tokens) + 3   # spread thin over the SMs, and ...
    trunk = build_trunk([128, 4, 2, 2, 1, 0])
    params = trunk_params(trunk)
    trunk = trunk.to(DEV)
    for B in (envs, 148 * (128 // tokens) + 1) if tokens in (5, 8, 17) else (envs,):   # ... tiles as full as they get
        x = torch.randn(B, tokens, 128, generator=gen)
        alive = torch.rand(B, tokens, generator=gen) < 0.7
        alive[0] = False
        hidden = torch.randn(2, B * tokens, 512, generator=gen) * 0.5
        ref_y, ref_h = O.trunk_step(x, alive, hidden, params, 4, "bf16")
        with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
            y, h = trunk.step(x.to(DEV), alive.to(DEV), hidden.to(DEV))
        assert_close(y, ref_y, "bf16", f"y, {B} environments")
        assert_close(h, ref_h, "bf16", f"hidden, {B} environments")
