"""Environments stay apart: one whose tokens or state are not finite leaves every other environment of the batch as it is in a
call without them, also where environments share an attention block (up to 8 tokens)."""

import pytest
import torch

from oracle import trunk_oracle as O
from tests.helpers import assert_close, build_trunk, trunk_params

pytestmark = pytest.mark.gpu
DEV = "cuda"
SIZES = [1, 2, 3, 5, 7, 8, 9, 12]   # the last two: an environment to a block


def poisoned(gen, lead, tokens, ships):
    """Tokens and state; the same with three bad environments (NaN tokens, an infinite one, a NaN state); the good environments."""
    B = lead[-1]
    x = torch.randn(*lead, tokens, 128, generator=gen)
    hidden = torch.randn(2, B * ships, 512, generator=gen) * 0.5
    bad = (1, 6, B - 2)   # neighbours on both sides; in the last tile too
    bad_x, bad_hidden = x.clone(), hidden.clone()
    bad_x[..., bad[0], :, :] = float("nan")
    bad_x[..., bad[1], tokens - 1, 5] = float("inf")
    bad_hidden[:, bad[2] * ships] = float("nan")
    return x, hidden, bad_x.to(DEV), bad_hidden.to(DEV), torch.tensor([b for b in range(B) if b not in bad])


def compare(got, clean, ref, good, ships, what):
    """The good environments near the oracle, and as in the call without bad ones: taken one by one their softmax sums are float32
    sums in another order, whose last bits move a few bfloat16 roundings (a quarter of the tolerance)."""
    rows = (good[:, None] * ships + torch.arange(ships)).flatten()
    for i, (dim, at, name) in enumerate(((-3, good, "y"), (1, rows, "hidden"))):
        assert not torch.isfinite(got[i]).all()   # the bad ones are bad
        ours = got[i].cpu().index_select(dim, at)
        assert_close(ours, clean[i].cpu().index_select(dim, at), "bf16", f"{what}: {name}, bad ones or not", scale=0.25)
        assert_close(ours, ref[i].index_select(dim, at), "bf16", f"{what}: {name}")


@pytest.mark.parametrize("tokens", SIZES)
@pytest.mark.parametrize("full", [False, True])
def test_step(tokens, full):
    gen = torch.Generator().manual_seed(tokens)
    ships = tokens - (tokens in (3, 7))   # two sizes with a field
    B = (148 if full else 1) * (128 // tokens) + 5   # tiles of several blocks, or environments spread thin
    x, hidden, bad_x, bad_hidden, good = poisoned(gen, (B,), tokens, ships)
    trunk = build_trunk([128, 4, 2, 2, 1, 0])
    ref = O.trunk_step(x, None, hidden, trunk_params(trunk), 4, "bf16")
    trunk = trunk.to(DEV)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        clean = trunk.step(x.to(DEV), None, hidden.to(DEV))
        got = trunk.step(bad_x, None, bad_hidden)
    compare(got, clean, ref, good, ships, f"{B} x {tokens}")


@pytest.mark.parametrize("tokens", SIZES)
def test_sequence(tokens):
    gen = torch.Generator().manual_seed(100 + tokens)
    ships = tokens - (tokens in (3, 7))
    T, B = 6, 2 * (128 // tokens) + 5
    x, hidden, bad_x, bad_hidden, good = poisoned(gen, (T, B), tokens, ships)
    done = torch.rand(T, B, generator=gen) < 0.2
    trunk = build_trunk([128, 4, 2, 2, 1, 0])
    ref = O.trunk_sequence(x, None, hidden, done, trunk_params(trunk), 4, "bf16")
    trunk = trunk.to(DEV)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        clean = trunk.sequence(x.to(DEV), None, hidden.to(DEV), done.to(DEV))
        got = trunk.sequence(bad_x, None, bad_hidden, done.to(DEV))
    compare(got, clean, ref, good, ships, f"{T} x {B} x {tokens}")
