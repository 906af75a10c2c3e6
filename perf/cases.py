"""The calls whose speed matters to a user of this package, over the sizes they are made at.

Five families, all through the public modules:

    step      ``YemongTrunk.step``: one rollout step of the trunk on the packed recurrent state,
              bfloat16 autocast (rollouts, evaluation) or float32 (crossover runs), with or without
              bullets and the folded reset of finished environments
    ragged    ``YemongTrunk.step_ragged``: one step over fleets of different sizes
    sequence  ``YemongTrunk.sequence`` without gradients: a stored rollout re-evaluated
    train     ``YemongTrunk.sequence`` and its backward: the recurrent-PPO minibatch
    policy    ``YemongPolicy.get_action_and_value``: encoders, trunk, heads, pooling, action draw

Trunk dimensions are those of the package's ``workloads.rl_config()`` (d_model 128, 4 heads, two
blocks of S S T, the first spatial sublayer of each block reading bullets).
"""

from __future__ import annotations

import contextlib
import math

import torch

import boost_and_broadside_b200 as bnb
from boost_and_broadside_b200 import workloads

DEV = "cuda"
D = 128
SHIP_FEATURES, BULLET_FEATURES, PREDICTED = 66, 26, 10  # widths of the standard coordinators
VALUE_COMPONENTS, TEAM_VALUES = 11, (0, 1)


def listed() -> list[dict]:
    return [
        # A handful of games being watched or evaluated with the whole policy: latency.
        _policy("policy_16", envs=16, bullets=80),
        # The rollout of a training run: 4v4 with four fields and ten bullet slots per ship.
        _policy("policy_8192", envs=8192, bullets=80),
        # The trunk alone at the latency end: an evaluation batch in one wave of the chip.
        _step("step_16x12", envs=16),
        # The trunk's headline size; finished environments are reset inside the step.
        _step("step_8192x12", envs=8192, reset=True),
        # The same with bullet tokens cross-attended.
        _step("step_8192x12_bullets", envs=8192, bullets=80),
        # Zero-shot large fleets: 64 against 88 ships, up to 70 % casualties.
        _step("step_1024x152", envs=1024, ships=152, fields=0, alive=0.65),
        # A crossover run's trunk in float32, an odd fleet with fields.
        _step("step_fp32_96x37", envs=96, ships=33, fields=4, fp32=True),
        # Mixed fleets of 2 to 128 tokens in one batch.
        dict(name="ragged_16384", kind="ragged", envs=16384, max_tokens=128),
        # A whole stored rollout re-evaluated, episode boundaries inside.
        _sequence("sequence_32x4096x8", "sequence", steps=32, envs=4096),
        # Short odd rollouts with bullets, as an evaluation logs them.
        _sequence("sequence_5x67x11_bullets", "sequence", steps=5, envs=67, ships=9, fields=2, bullets=45),
        # A PPO minibatch, forward and backward.
        _sequence("train_32x1024x8", "train", steps=32, envs=1024),
        # A small minibatch of the profile with fields and bullets.
        _sequence("train_16x96x12_bullets", "train", steps=16, envs=96, fields=4, bullets=80),
    ]


def _step(name, envs, ships=8, fields=4, bullets=0, alive=0.9, reset=False, fp32=False):
    return dict(name=name, kind="step", envs=envs, ships=ships, fields=fields, bullets=bullets, alive=alive, reset=reset, fp32=fp32)


def _policy(name, envs, ships=8, fields=4, bullets=0):
    return dict(name=name, kind="policy", envs=envs, ships=ships, fields=fields, bullets=bullets)


def _sequence(name, kind, steps, envs, ships=8, fields=0, bullets=0):
    return dict(name=name, kind=kind, steps=steps, envs=envs, ships=ships, fields=fields, bullets=bullets)


def draw(rng) -> dict:
    """One more case of a random family.  Fleets of 2 to 152 ships (small ones mostly, as in use), 0
    to 4 fields, bullets in half the cases, environments over the logarithm of what the family holds."""
    kind = rng.choice(("step", "step", "step_fp32", "ragged", "sequence", "train", "policy"))

    def log(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(max(lo, hi) + 0.5))))))

    if kind == "ragged":
        return dict(kind="ragged", envs=log(16, 12000), max_tokens=rng.randint(12, 128))
    large = kind in ("step", "step_fp32") and rng.random() < 0.3
    ships = rng.randint(17, 152) if large else log(2, 24 if kind in ("step", "sequence", "policy") else 16)
    fields = rng.choice((0, rng.randint(1, 4)))
    bullets = rng.choice((0, min(160, ships * rng.randint(1, 10))))
    tokens = ships + fields
    if kind == "step":
        case = _step("", log(1, 131072 // (tokens + bullets // 8)), ships, fields, bullets, rng.uniform(0.5, 1.0), rng.random() < 0.5)
    elif kind == "step_fp32":
        case = _step("", log(1, 16384 // (tokens + bullets // 2)), ships, fields, bullets, rng.uniform(0.5, 1.0), False, True)
    elif kind == "policy":
        case = _policy("", log(1, 98304 // (tokens + bullets // 8)), ships, fields, bullets)
    else:
        steps = log(2, 64)
        rows = 524288 if kind == "sequence" else 131072
        case = _sequence("", kind, steps, log(1, rows // (steps * (tokens + bullets))), ships, fields, bullets)
    del case["name"]
    return case


# ----------------------------------------------------------------------------- inputs


def _model(make, seed: int):
    """A module with its own seeded initialisation, its norm gains and near-zero parameters moved off
    their initial values as training moves them."""
    with torch.random.fork_rng(devices=[]):
        torch.manual_seed(seed)
        model = make()
        with torch.no_grad():
            for name, p in model.named_parameters():
                if name.endswith("seeds"):
                    p.normal_(0.0, 0.5)
                elif p.dim() == 1 and bool((p == 1).all()):
                    p.add_(0.1 * torch.randn_like(p))
                elif "field_sub" in name:
                    p.add_(0.02 * torch.randn_like(p))
    return model.to(DEV)


def _alive(gen, lead: tuple, ships: int, fields: int, p: float) -> torch.Tensor:
    """Ships alive with probability p, one per team at least; fields always."""
    alive = torch.rand(*lead, ships, device=DEV, generator=gen) < p
    alive[..., 0] = True
    alive[..., ships // 2] = True
    return torch.cat([alive, torch.ones(*lead, fields, dtype=torch.bool, device=DEV)], dim=-1)


def _in_flight(gen, envs: int, slots: int) -> torch.Tensor:
    """Bullet slots in use: about 30 %, and none at all in a quarter of the environments."""
    mask = torch.rand(envs, slots, device=DEV, generator=gen) < 0.3
    return mask & (torch.rand(envs, 1, device=DEV, generator=gen) >= 0.25)


def _hidden(gen, rows: int) -> torch.Tensor:
    return torch.randn(2, rows, 4 * D, device=DEV, generator=gen) * 0.5


class _Observation(dict):
    """What the caller's environment hands the policy: per-token channels and a dict of bullet channels."""

    bullets = None


class _Coordinator:
    """The caller's feature coordinator; the raw feature vectors are ready in the observation."""

    total_prediction_dimension = PREDICTED

    def __init__(self, width: int, read) -> None:
        self.total_input_dimension = width
        self.get_input_vector = read


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device=DEV).manual_seed(seed)
    state = dict(case=case, kind=case["kind"])
    if case["kind"] == "ragged":
        return _prepare_ragged(case, seed, gen, state)
    envs, ships, fields, slots = case["envs"], case["ships"], case["fields"], case["bullets"]
    steps = case.get("steps")
    lead = (envs,) if steps is None else (steps, envs)
    state["alive"] = _alive(gen, lead, ships, fields, case.get("alive", 0.9))
    state["hidden"] = _hidden(gen, envs * ships)
    if case["kind"] == "policy":
        obs = _Observation(alive=state["alive"], raw=torch.rand(envs, ships + fields, SHIP_FEATURES, device=DEV, generator=gen) * 2 - 1,
                           team_id=(torch.arange(ships + fields, device=DEV) * 2 // ships).clamp(max=1).expand(envs, -1).contiguous())
        if slots:
            obs.bullets = {"raw": torch.rand(envs, slots, BULLET_FEATURES, device=DEV, generator=gen) * 2 - 1,
                           "ACTIVE": _in_flight(gen, envs, slots)}
        state.update(obs=obs, gen=torch.Generator(device=DEV).manual_seed(seed + 1))
        state["policy"] = _model(lambda: bnb.YemongPolicy(
            workloads.rl_config(), _Coordinator(SHIP_FEATURES, lambda o: o["raw"]), VALUE_COMPONENTS, ships, TEAM_VALUES,
            bullet_coordinator=_Coordinator(BULLET_FEATURES, lambda o: o.bullets["raw"])).eval(), seed)
        return state
    # The tokens an encoder under bfloat16 autocast hands the trunk are bfloat16.
    dtype = torch.float32 if case.get("fp32") else torch.bfloat16
    state["x"] = torch.randn(*lead, ships + fields, D, device=DEV, generator=gen).to(dtype)
    state["bullets"], state["mask"] = None, None
    if slots:
        state["bullets"] = torch.randn(math.prod(lead), slots, D, device=DEV, generator=gen).to(dtype)
        state["mask"] = _in_flight(gen, math.prod(lead), slots)
    if steps is None:
        state["reset"] = torch.rand(envs, device=DEV, generator=gen) < 0.02 if case["reset"] else None
    else:
        state["done"] = torch.rand(steps, envs, device=DEV, generator=gen) < 0.02
    state["trunk"] = _model(lambda: bnb.YemongTrunk(workloads.rl_config()), seed)
    if case["kind"] == "train":
        state["x"].requires_grad_(True)
        if slots:
            state["bullets"].requires_grad_(True)
        state["dy"] = (torch.randn(state["x"].shape, device=DEV, generator=gen) / state["x"].numel() ** 0.5).to(dtype)
        # A field-free batch leaves the field substitute out of the graph, as in the reference.
        state["params"] = [p for n, p in state["trunk"].named_parameters() if fields or "field_sub" not in n]
        if not slots:
            unused = {id(p) for n, p in state["trunk"].named_parameters() if "_bullet" in n}
            state["params"] = [p for p in state["params"] if id(p) not in unused]
    return state


def _prepare_ragged(case: dict, seed: int, gen, state: dict) -> dict:
    # An even spread of sizes in a random order, so that a batch of another seed has as many rows.
    order = torch.randperm(case["envs"], generator=torch.Generator().manual_seed(seed))
    tokens = 2 + order * (case["max_tokens"] - 1) // case["envs"]
    fields = torch.minimum(order % 5, tokens - 2)
    ships = tokens - fields
    total = int(tokens.sum())
    state["ragged"] = bnb.RaggedBatch(tokens, ships)
    state["x"] = torch.randn(total, D, device=DEV, generator=gen).to(torch.bfloat16)
    first = (tokens.cumsum(0) - tokens).to(DEV)
    alive = torch.rand(total, device=DEV, generator=gen) < 0.9
    alive[first] = True
    state["alive"] = alive
    state["hidden"] = _hidden(gen, int(ships.sum()))
    state["trunk"] = _model(lambda: bnb.YemongTrunk(workloads.rl_config()), seed)
    return state


# ----------------------------------------------------------------------------- one pass


def run(state: dict):
    case, kind = state["case"], state["kind"]
    autocast = contextlib.nullcontext() if case.get("fp32") else torch.autocast("cuda", dtype=torch.bfloat16)
    if kind == "train":
        with autocast:
            y, hidden = state["trunk"].sequence(state["x"], state["alive"], state["hidden"], state["done"],
                                                bullets=state["bullets"], bullet_mask=state["mask"])
        inputs = [state["x"]] + ([] if state["bullets"] is None else [state["bullets"]])
        grads = torch.autograd.grad(y, inputs + state["params"], state["dy"])
        # One vector of all parameter gradients, as norm clipping and flat optimizers take them.
        flat = torch.cat([g.reshape(-1) for g in grads[len(inputs):]])
        return (y.detach(), hidden.detach(), *grads[: len(inputs)], flat)
    with torch.no_grad(), autocast:
        if kind == "policy":
            return state["policy"].get_action_and_value(state["obs"], state["hidden"], generator=state["gen"])
        if kind == "ragged":
            return state["trunk"].step_ragged(state["x"], state["alive"], state["hidden"], state["ragged"])
        if kind == "step":
            return state["trunk"].step(state["x"], state["alive"], state["hidden"], reset_env=state["reset"],
                                       bullets=state["bullets"], bullet_mask=state["mask"])
        return state["trunk"].sequence(state["x"], state["alive"], state["hidden"], state["done"],
                                       bullets=state["bullets"], bullet_mask=state["mask"])


# ----------------------------------------------------------------------------- work and tolerance


def work(case: dict) -> dict:
    """Two operations per multiply-add: a spatial sublayer 16 D^2 per token and 2 D per query and key, a
    temporal one 17 D^2 per ship and 16 D^2 per field; four spatial and two temporal sublayers, two of the
    spatial ones reading the bullets in flight (22 % of the slots).  Bytes: tokens, bullets, masks and
    state in, tokens and state out, each once, parameters once in float32."""
    steps = case.get("steps", 1)
    if case["kind"] == "ragged":
        n = (case["max_tokens"] + 2) / 2
        tokens, fields = case["envs"] * n, case["envs"] * 2.0
        pairs = case["envs"] * sum(k * k for k in range(2, case["max_tokens"] + 1)) / (case["max_tokens"] - 1)
        ships, states, bullets, slots = tokens - fields, tokens - fields, 0, 0
    else:
        n = case["ships"] + case["fields"]
        calls = case["envs"] * steps
        tokens, ships, fields, states = calls * n, calls * case["ships"], calls * case["fields"], case["envs"] * case["ships"]
        slots = calls * case["bullets"]
        bullets, pairs = 0.225 * slots, tokens * n
    flops = 4 * (2 * 16 * D * D * tokens + 4 * D * pairs) + 2 * 2 * D * D * (17 * ships + 16 * fields)
    if slots:
        flops += 2 * (2 * 2 * D * D * bullets + 4 * D * tokens * bullets / slots * case["bullets"])
    size = 4 if case.get("fp32") else 2
    bytes_ = 2 * size * D * tokens + tokens + 2 * 2 * 4 * 4 * D * states + 4 * 1.71e6
    bytes_ += size * D * bullets + slots
    if case["kind"] == "train":
        flops *= 3
        bytes_ += 2 * size * D * tokens + 2 * size * D * slots + 4 * 1.71e6
    if case["kind"] == "policy":
        hidden, bullet_hidden = 2 * D, 64
        flops += 2 * tokens * hidden * (SHIP_FEATURES + D) + 2 * bullets * bullet_hidden * (BULLET_FEATURES + D)
        flops += 2 * ships * (4 * hidden * D + hidden * (12 + VALUE_COMPONENTS + len(TEAM_VALUES) + PREDICTED) + 2 * D * D)
        bytes_ -= 2 * size * D * tokens + size * D * bullets  # tokens stay inside
        bytes_ += 4 * (SHIP_FEATURES * tokens + BULLET_FEATURES * bullets) + ships * (24 + 2 * (1 + VALUE_COMPONENTS + PREDICTED))
    return {"bytes": bytes_, "flops": flops}


def tolerance(case: dict):
    """float32 sums through six sublayers; bfloat16 operands everywhere else, whose gradients go through
    twice the roundings.  An action draw may fall on the other side of a boundary moved by a rounding."""
    if case.get("fp32"):
        return {"rel": 2e-5, "max": 1e-3}
    if case["kind"] == "train":
        return {"rel": 2e-2, "max": 0.5}
    if case["kind"] == "policy":
        return {"rel": 1e-2, "max": 0.5, "differ": 0.01}
    return {"rel": 1e-2, "max": 0.3}
