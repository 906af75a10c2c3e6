"""Inference outputs that have no sums in an order of chance, bit for bit as recorded (golden/recorded_bits.json, digests).  The order
of a float32 sum is part of these results: another one moves bfloat16 roundings in every sublayer behind it, the float32 recurrent
state by 1e-4 and a few of the actions drawn from the same random numbers."""

import hashlib
import json
import os

import pytest
import torch

from tests.helpers import GOLDEN, build_trunk
from tests.test_gpu_policy_tail import _Obs, _policy

pytestmark = pytest.mark.gpu
DEV = "cuda"

# tokens, bullet slots, share of them in use (None: no mask): one and several blocks of queries, of keys, of bullet rows
STEPS = [(12, 80, 0.3), (12, 80, None), (16, 33, 0.5), (5, 16, 0.6), (3, 160, 0.9), (33, 100, 0.5), (129, 0, 0.0), (152, 0, 0.0)]
# environments, ships, fields, bullet slots: one row tile and several, the encoder of wanted rows and of all
POLICIES = [(16, 8, 0, 0), (300, 8, 4, 80), (41, 5, 1, 33), (700, 2, 0, 0)]
# steps, environments, ships, fields, bullet slots, share of them in use (None: no mask), autocast
TRAINS = [(5, 3, 4, 1, 0, 0.0, 1), (9, 3, 12, 4, 80, 0.3, 1), (2, 3, 8, 0, 100, 0.7, 1), (2, 3, 8, 0, 40, None, 1), (2, 2, 20, 3, 90, 0.6, 1), (3, 2, 30, 0, 0, 0.0, 1),
          (4, 3, 7, 2, 70, 0.6, 0), (33, 40, 3, 0, 0, 0.0, 1)]


def digest(*tensors) -> str:
    h = hashlib.sha256()
    for t in tensors:
        h.update(t.detach().cpu().contiguous().view(torch.uint8).numpy().tobytes())
    return h.hexdigest()[:24]


def step_digest(tokens, slots, share) -> str:
    gen = torch.Generator().manual_seed(1000 * tokens + slots)
    envs = 9
    trunk = build_trunk([128, 4, 2, 2, 1, 1]).to(DEV)
    x = torch.randn(envs, tokens, 128, generator=gen).to(DEV, torch.bfloat16)
    alive = (torch.rand(envs, tokens, generator=gen) < 0.8).to(DEV)
    hidden = (torch.randn(2, envs * tokens, 512, generator=gen) * 0.5).to(DEV)
    bullets = torch.randn(envs, slots, 128, generator=gen).to(DEV, torch.bfloat16) if slots else None
    mask = (torch.rand(envs, slots, generator=gen) < share).to(DEV) if slots and share is not None else None
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        return digest(*trunk.step(x, alive, hidden, bullets=bullets, bullet_mask=mask))


def policy_digest(envs, ships, fields, slots) -> str:
    p = _policy(ships, seed=envs)
    gen = torch.Generator().manual_seed(envs + slots)
    obs = _Obs(alive=(torch.rand(envs, ships + fields, generator=gen) < 0.8).to(DEV), raw=torch.randn(envs, ships + fields, 66, generator=gen).to(DEV),
               team_id=torch.randint(0, 2, (envs, ships + fields), generator=gen).to(DEV))
    obs.bullets = {"raw": torch.randn(envs, slots, 26, generator=gen).to(DEV), "ACTIVE": (torch.rand(envs, slots, generator=gen) < 0.3).to(DEV)} if slots else None
    hidden = (torch.randn(2, envs * ships, 512, generator=gen) * 0.5).to(DEV)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        every = p.bullet_encoder.encode_raw(obs.bullets["raw"]) if slots else hidden   # in steps alone the slots in use are encoded
        return digest(every, *p.get_action_and_value(obs, hidden, torch.Generator(device=DEV).manual_seed(3)))


def train_digest(steps, envs, ships, fields, slots, share, autocast) -> str:
    """Results and the gradients that belong to one row; those of parameters are summed by atomics (and so is d q beyond 32 tokens)."""
    gen = torch.Generator().manual_seed(100 * steps + ships + slots)
    trunk = build_trunk([128, 4, 2, 2, 1, 1]).to(DEV)
    half = torch.bfloat16 if autocast else torch.float32
    x = torch.randn(steps, envs, ships + fields, 128, generator=gen).to(DEV, half).requires_grad_()
    alive = (torch.rand(steps, envs, ships + fields, generator=gen) < 0.8).to(DEV)
    hidden = (torch.randn(2, envs * ships, 512, generator=gen) * 0.5).to(DEV).requires_grad_()
    done = (torch.rand(steps, envs, generator=gen) < 0.2).to(DEV)
    bullets = torch.randn(steps * envs, slots, 128, generator=gen).to(DEV, half).requires_grad_() if slots else None
    mask = (torch.rand(steps * envs, slots, generator=gen) < share).to(DEV) if slots and share is not None else None
    dy, dh = torch.randn(x.shape, generator=gen).to(DEV, half), torch.randn(hidden.shape, generator=gen).to(DEV)
    with torch.autocast(DEV, dtype=torch.bfloat16, enabled=bool(autocast)):
        y, h = trunk.sequence(x, alive, hidden, done, bullets=bullets, bullet_mask=mask)
    rows = [x, hidden] + ([bullets] if slots else [])
    return digest(y, h, *torch.autograd.grad([y, h], rows, [dy, dh]))


def recorded() -> dict:
    with open(os.path.join(GOLDEN, "recorded_bits.json")) as f:
        return json.load(f)


@pytest.mark.parametrize("tokens,slots,share", STEPS)
def test_step(tokens, slots, share):
    assert step_digest(tokens, slots, share) == recorded()[f"step {tokens} {slots} {share}"]


@pytest.mark.parametrize("envs,ships,fields,slots", POLICIES)
def test_policy(envs, ships, fields, slots):
    assert policy_digest(envs, ships, fields, slots) == recorded()[f"policy {envs} {ships} {fields} {slots}"]


@pytest.mark.parametrize("mode", ["keep", "recompute"])
@pytest.mark.parametrize("steps,envs,ships,fields,slots,share,autocast", TRAINS)
def test_train(steps, envs, ships, fields, slots, share, autocast, mode, monkeypatch):
    monkeypatch.setenv("BNB_GRAD_MODE", mode)
    assert train_digest(steps, envs, ships, fields, slots, share, autocast) == recorded()[f"train {mode} {steps} {envs} {ships} {fields} {slots} {share} {autocast}"]
