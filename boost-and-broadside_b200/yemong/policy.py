"""The rollout step of the policy on CUDA kernels end to end, mirroring ``YemongPolicy`` of the
reference (models/yemong/policy.py:135-373).

``YemongPolicy`` here has the reference's constructor arguments, sub-module names and parameter
names (``encoder``, ``bullet_encoder``, ``yemong_layers``, ``action_head``, ``value_head_local``,
``team_pma``, ``value_head_win``, ``next_state_head``), so a reference ``state_dict`` loads
unchanged.  ``get_action_and_value`` (policy.py:291-373) runs, from the coordinators' raw feature
vectors on: the encoder kernels, the trunk in one call on the packed state, the head kernels,
TeamPMA and the action draw.  The ``FeatureCoordinator`` objects are the caller's and run as they
are.  ``evaluate_actions`` (policy.py:379-516) is mirrored as a forward: evaluation, crossover and
logging call it without gradients.  For the PPO update itself -- ``evaluate_actions`` differentiated
-- keep the reference's policy and swap its blocks for this package's ``YemongBlock``: the trunk then
runs forward and backward here, and the reference's encoders and heads, which have no backward in
this package, stay torch modules.
"""

from __future__ import annotations

import torch
import torch.nn as nn

from .. import _capi
from . import _end_ops, _ops
from .encoder import BulletEncoder, ShipEncoder
from .griffin import YemongBlock
from .heads import HeadMLP, NextStateHead, TeamPMA, evaluate_action, sample_action
from .trunk import YemongTrunk

TOTAL_ACTION_LOGITS = 12  # constants.py:43


# Queries of the library about sizes: constants of a trace.
@torch.compiler.assume_constant_result
def _bullets_compacted(d_model: int, n_heads: int, n_tokens: int, n_slots: int) -> bool:
    return _capi.host.bullets_compacted(d_model, n_heads, n_tokens, n_slots)


@torch.compiler.assume_constant_result
def _tail_supported(d_model: int, n_heads: int, n_ships: int, *head_widths: int) -> bool:
    return _capi.host.tail_supported(d_model, n_heads, n_ships, list(head_widths))


def _plain(module: nn.Module, cls: type) -> bool:
    """Whether calling ``module`` is what ``cls.forward`` does: no subclass's forward, no hooks."""
    return (type(module) is cls and not module._forward_hooks and not module._forward_pre_hooks
            and not torch.nn.modules.module._has_any_global_hook())


class YemongPolicy(YemongTrunk):
    """Encoder -> n x YemongBlock -> heads (policy.py:135-214), rollout path."""

    def __init__(self, model_config, coordinator, num_value_components: int, num_ships: int,
                 team_pma_k: tuple[int, ...], bullet_coordinator=None) -> None:
        nn.Module.__init__(self)   # sub-modules are registered below in the reference's order
        D = model_config.d_model
        self.d_model = self._d_model = D
        self.n_heads = model_config.n_heads
        self.n_temporal = self._n_temporal = model_config.n_temporal_per_block
        self._K = num_value_components
        self._num_ships = num_ships
        self._team_pma_k = tuple(team_pma_k)
        self.coordinator = coordinator
        self.encoder = ShipEncoder(model_config, coordinator, num_ships=num_ships)
        self.bullet_encoder = (BulletEncoder(model_config, bullet_coordinator)
                               if model_config.reads_bullets and bullet_coordinator is not None else None)
        self.yemong_layers = nn.ModuleList([YemongBlock(model_config) for _ in range(model_config.n_yemong_blocks)])
        self.action_head = HeadMLP(D, TOTAL_ACTION_LOGITS)
        self.value_head_local = HeadMLP(D, num_value_components)
        if self._team_pma_k:
            self.team_pma = TeamPMA(D, model_config.n_heads)
            self.value_head_win = HeadMLP(D, len(self._team_pma_k))
        self.next_state_head = NextStateHead(D, coordinator.total_prediction_dimension)

    @property
    def num_recurrent_tokens(self) -> int:
        return self._num_ships

    def _encode_bullets(self, obs, n_tokens: int):
        """Bullet tokens and their mask.  The trunk's tensor-core kernels read the tokens of active slots
        only, so where they serve the call (environments of ``n_tokens``) the others are not encoded."""
        enc = self.bullet_encoder
        if enc is None or obs.bullets is None:
            return None, None
        active = next(v for k, v in obs.bullets.items() if getattr(k, "name", str(k)).upper().endswith("ACTIVE"))
        if not _plain(enc, BulletEncoder):
            return enc(obs), active
        raw = enc.coordinator.get_input_vector(obs)
        compacts = (_capi.current_precision(raw.device) == _capi.BNB_BF16 and tuple(active.shape) == tuple(raw.shape[:-1])
                    and _bullets_compacted(self.d_model, self.n_heads, n_tokens, raw.shape[-2]))
        return enc.encode_raw(raw, active if compacts else None), active

    def _tail_lists(self):
        """Parameters of the heads and of TeamPMA as ``_end_ops.policy_tail`` takes them, or None where
        its kernels do not serve this policy (modules of other widths, replaced ones, ones with hooks)."""
        if not _plain(self.next_state_head, NextStateHead):
            return None
        heads = [self.action_head, self.next_state_head.net, self.value_head_local]
        pma: list[torch.Tensor] = []
        if self._team_pma_k:
            heads.append(self.value_head_win)
            if not _plain(self.team_pma, TeamPMA) or self.team_pma.n_heads != self.n_heads or self.team_pma.d_model != self.d_model:
                return None
            pma = [self.team_pma.seeds, self.team_pma.attn.in_proj_weight, self.team_pma.attn.out_proj.weight, self.team_pma.norm.weight]
        if not all(_plain(h, HeadMLP) for h in heads):
            return None
        lists = [h.parameter_list() for h in heads]
        if not _tail_supported(self.d_model, self.n_heads, self._num_ships,
                               *[w for ps in lists for w in (ps[0].shape[1], ps[0].shape[0], ps[3].shape[0])]):
            return None
        return [p for ps in lists for p in ps], pma

    @torch.no_grad()
    def get_action_and_value(self, obs, hidden: torch.Tensor, generator: torch.Generator | None = None):
        """One rollout step (policy.py:291-373): returns (action (B, N, 3), logprob (B, N),
        value (B, N, K), pred_next (B, N, pred_dim), new_hidden)."""
        alive = obs["alive"]
        x = self.encoder(obs)
        bullets, bullet_mask = self._encode_bullets(obs, x.shape[1])
        x, new_hidden = self.step(x, alive, hidden, bullets=bullets, bullet_mask=bullet_mask)
        N = self._num_ships
        lists = self._tail_lists() if x.dtype == torch.bfloat16 and x.shape[1] >= N else None
        if lists is not None:
            uniforms = torch.rand(x.shape[0] * N, 3, device=x.device, generator=generator)
            run = _capi.host.policy_tail if _ops.direct(x) else _end_ops.policy_tail
            teams = (alive, obs["team_id"]) if self._team_pma_k else (None, None)
            action, logprob, value, pred_next = run(x, *teams, uniforms, *lists, list(self._team_pma_k), N)
            return action, logprob, value, pred_next, new_hidden
        x_ships = x[:, :N, :].contiguous()
        logits = self.action_head(x_ships)
        pred_next = self.next_state_head(x_ships)
        value = self.value_head_local(x_ships)
        if self._team_pma_k:
            x_team = self.team_pma(x_ships, obs["team_id"][:, :N], alive[:, :N])
            win_val = self.value_head_win(x_team)
            for i, k in enumerate(self._team_pma_k):
                value[:, :, k] = win_val[:, :, i]
        action, logprob = sample_action(logits, generator)
        return action, logprob, value, pred_next, new_hidden

    @torch.no_grad()
    def evaluate_actions(self, obs, actions: torch.Tensor, initial_hidden: torch.Tensor, alive_mask: torch.Tensor,
                         done_mask: torch.Tensor | None = None, return_encoder_output: bool = False):
        """The rollout re-evaluated over T steps (policy.py:379-516), without gradients: obs with
        (T, B, N+M, ...) tensors, actions (T, B, N, 3).  Returns (logprob (T, B, N), entropy (T, B, N),
        value (T, B, N, K), logits (T, B, N, 12), encoder output or None, pred_next (T, B, N, pred_dim))."""
        T, B, N = actions.shape[:3]
        flat = type(obs)(
            data={k: v.reshape(T * B, *v.shape[2:]) for k, v in obs.items()},
            bullets=None if obs.bullets is None else {k: v.reshape(T * B, *v.shape[2:]) for k, v in obs.bullets.items()},
        )
        x = self.encoder(flat)
        NM, D = x.shape[1], x.shape[2]
        x = x.reshape(T, B, NM, D)
        bullets, bullet_mask = self._encode_bullets(flat, NM)
        z = x if return_encoder_output else None
        x, _ = self.sequence(x, alive_mask, initial_hidden, done_mask, bullets=bullets, bullet_mask=bullet_mask)
        x_ships = x[:, :, :N, :].contiguous()
        logits = self.action_head(x_ships)
        pred_next = self.next_state_head(x_ships)
        value = self.value_head_local(x_ships)
        if self._team_pma_k:
            pooled = self.team_pma(x_ships.reshape(T * B, N, D), obs["team_id"][:, :, :N].reshape(T * B, N),
                                   alive_mask[:, :, :N].reshape(T * B, N))
            win_val = self.value_head_win(pooled.reshape(T, B, N, D))
            for i, k in enumerate(self._team_pma_k):
                value[..., k] = win_val[..., i]
        logprob, entropy = evaluate_action(logits, actions)
        return logprob, entropy, value, logits, z, pred_next
