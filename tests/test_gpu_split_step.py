"""The float32 step on tensor-core tiles: tile edges, every split of columns and hidden chunks over CTAs, fleets
above one attention chunk, bullet rings above one slot pass, against the CPU oracle or, where that takes long,
the exact kernels."""

from __future__ import annotations

import pytest
import torch

from oracle import trunk_oracle as O
from tests.helpers import assert_close, build_trunk, trunk_params

pytestmark = pytest.mark.gpu
DEV = "cuda"


# rows: 1, 127, 128, 129; 18 | 19, 37 | 38 and 74 | 75 tiles are where the splits change, 151 is above one wave
@pytest.mark.parametrize("B,N,M,NB", [(1, 1, 0, 0), (127, 1, 0, 1), (32, 4, 0, 0), (43, 2, 1, 5), (3, 16, 0, 16), (2, 17, 0, 17),
                                      (2, 31, 2, 128), (3, 60, 4, 129), (1, 152, 4, 300), (192, 8, 4, 0), (193, 8, 4, 3), (394, 8, 4, 0),
                                      (400, 8, 4, 20), (789, 8, 4, 0), (798, 8, 4, 2), (1600, 8, 4, 33), (9, 0, 5, 4)])
def test_float32_step_on_tiles(B, N, M, NB):
    from boost_and_broadside_b200 import _capi

    g = torch.Generator().manual_seed(B * 7 + N)
    x = torch.randn(B, N + M, 128, generator=g)
    alive = torch.rand(B, N + M, generator=g) < 0.7
    alive[0] = False
    hidden = torch.randn(2, B * N, 512, generator=g) * 0.5
    reset = torch.rand(B, generator=g) < 0.3
    bul = torch.randn(B, NB, 128, generator=g) if NB else None
    mask = torch.rand(B, NB, generator=g) < 0.3 if NB else None
    if NB:
        mask[B // 2] = False
    trunk = build_trunk([128, 4, 2, 2, 1, 1])
    move = lambda t: None if t is None else t.to(DEV)  # noqa: E731
    small = B * (N + M) < 1000
    if small:
        ref = O.trunk_step(x, alive, O.reset_hidden_for_envs(hidden, reset, N), trunk_params(trunk), 4, "fp32", bul, mask)
    trunk = trunk.to(DEV)
    with torch.no_grad():
        args = (move(x), move(alive), move(hidden), move(reset))
        got = trunk.step(*args, bullets=move(bul), bullet_mask=move(mask))
        if not small:
            ref = trunk.step(*args, engine=_capi.ENGINE_SIMT, bullets=move(bul), bullet_mask=move(mask))
    assert_close(got[0], ref[0], "fp32", "y")
    if N:
        assert_close(got[1], ref[1], "fp32", "hidden")
