"""A sequence's temporal sublayers on tiles of several timesteps per token (pipelined_tile_kernel.cu, STEPS) against the
oracle: every chunk length, sequences shorter than, equal to and longer than a chunk, a last tile that is not full, fields,
episode boundaries at every lag, and the walk over tiles of one timestep where the rule keeps it."""

import pytest
import torch

from tests.helpers import assert_close, build_trunk, trunk_params
from oracle import trunk_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"

CASES = [
    # T, environments, ships, fields
    (2, 3, 5, 0),        # chunks of 4, half of each empty
    (4, 7, 8, 4),        # one full chunk of 4
    (5, 67, 9, 2),       # 8
    (8, 1, 1, 0),        # 8, one token
    (13, 3, 2, 3),       # 16
    (17, 5, 8, 4),       # 32
    (33, 9, 8, 0),       # 32, two chunks, one step in the second
    (33, 70, 10, 0),     # 16, three chunks
    (20, 600, 8, 0),     # 8: more tiles than SMs
    (7, 2, 100, 52),     # environments larger than a tile
    (2, 2368, 8, 0),     # the walk: two steps of a batch that fills the chip
    (3, 2365, 8, 0),     # the walk, a last tile that is not full
    (5, 1475, 8, 4),     # the walk with fields
    (4, 2368, 8, 0),     # as many passes in chunks of 4
]


@pytest.mark.parametrize("T,B,ships,fields", CASES)
@pytest.mark.parametrize("token_dtype", [torch.float32, torch.bfloat16])
def test_chunked_sequence_against_the_oracle(T, B, ships, fields, token_dtype):
    gen = torch.Generator().manual_seed(1000 * T + B)
    N = ships + fields
    x = torch.randn(T, B, N, 128, generator=gen).to(token_dtype)
    alive = torch.rand(T, B, N, generator=gen) < 0.8
    alive[..., 0] = True
    hidden = torch.randn(2, B * ships, 512, generator=gen) * 0.5
    done = torch.rand(T, B, generator=gen) < 0.3
    trunk = build_trunk([128, 4, 2, 2, 1, 0])
    ref_y, ref_h = O.trunk_sequence(x.float(), alive, hidden, done, trunk_params(trunk), 4, "bf16")
    trunk = trunk.to(DEV)
    given = hidden.to(DEV)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        y, nh = trunk.sequence(x.to(DEV), alive.to(DEV), given, done.to(DEV))
    torch.cuda.synchronize()
    # bfloat16 tokens: one more rounding of the stream where a launch hands over (four launches)
    assert_close(y, ref_y, "bf16", "y")
    assert_close(nh, ref_h, "bf16", "hidden")
    assert torch.equal(given.cpu(), hidden)   # the caller's state is not written


def test_a_sequence_continues_where_the_one_before_ended():
    """Taps and state across calls: 12 steps at once against 5 and 7, whose chunks sum the recurrence in another order: equal to a
    quarter of the tolerance (a float32 sum's last bit, and the bfloat16 roundings it moves)."""
    gen = torch.Generator().manual_seed(5)
    x = torch.randn(12, 6, 8, 128, generator=gen).to(DEV)
    done = (torch.rand(12, 6, generator=gen) < 0.2).to(DEV)
    done[4] = False   # a flag of a call's last step is the caller's to apply
    hidden = (torch.randn(2, 48, 512, generator=gen) * 0.5).to(DEV)
    trunk = build_trunk([128, 4, 2, 2, 1, 0]).to(DEV)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        y, h = trunk.sequence(x, None, hidden, done)
        ya, ha = trunk.sequence(x[:5], None, hidden, done[:5])
        yb, hb = trunk.sequence(x[5:], None, ha, done[5:])
    # lags right after the cut look at stored taps in one call and at rows above in the other: same values unless an episode
    # began within the last two steps, whose flags the second call does not see
    fresh = ~(done[2:4].any(0))
    assert_close(torch.cat([ya, yb])[:, fresh], y[:, fresh], "bf16", "y", scale=0.25)
    rows = fresh.repeat_interleave(8)
    assert_close(hb[:, rows], h[:, rows], "bf16", "hidden", scale=0.25)
