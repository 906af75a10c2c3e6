"""Opaque ``torch.library`` operators for the ends of the policy step: the encoder / head MLP
chain, TeamPMA and the action distribution.

Same reason as ``_ops.py``: ``torch.compile(policy.get_action_and_value, mode="reduce-overhead")``
(how the reference runs its policy, train/rl/ppo.py:396-400) must see one opaque node per call
into the C ABI, with a shape-only fake implementation, so that the FeatureCoordinator's torch
operators around them are fused by the compiler and the whole step replays as one CUDA graph.
All of them are forward-only.
"""

from __future__ import annotations

from typing import List, Optional, Tuple

import torch
from torch import Tensor

from .. import _capi


def _out_dtype(precision: int) -> torch.dtype:
    return torch.bfloat16 if precision == _capi.BNB_BF16 else torch.float32


def _check_params(dev: torch.device, what: str, *ps: Optional[Tensor]) -> None:
    for p in ps:
        if p is not None and (p.device != dev or p.dtype != torch.float32 or not p.is_contiguous()):
            raise RuntimeError(f"{what} parameters must be contiguous float32 on the input's device")


@torch.library.custom_op("bnb_b200::mlp_chain", mutates_args=(), device_types="cuda")
def mlp_chain(x: Tensor, w1: Tensor, b1: Tensor, g1: Tensor, w2: Tensor, b2: Tensor, g2: Optional[Tensor],
              precision: int, active: Optional[Tensor] = None) -> Tensor:
    """Linear(w1, b1) -> RMSNorm(g1) -> GELU -> Linear(w2, b2) [-> RMSNorm(g2)] over the rows of
    x (rows, in): with g2 the encoders, without it the heads.  Returns (rows, out), bfloat16 under the
    bfloat16 contract, else float32.  ``active`` (rows,) bool: the caller uses only these rows of the
    result; where the tiled kernel serves the call the others are not computed and hold anything."""
    return mlp_call(x, w1, b1, g1, w2, b2, g2, precision, active)


def mlp_call(x, w1, b1, g1, w2, b2, g2, precision, active=None):
    """The body of ``mlp_chain``, in native code (csrc/host_path.cpp)."""
    return _capi.host.mlp_chain(x, [w1, b1, g1, w2, b2] if g2 is None else [w1, b1, g1, w2, b2, g2], precision, active)


@mlp_chain.register_fake
def _(x, w1, b1, g1, w2, b2, g2, precision, active=None):
    return x.new_empty((x.shape[0], w2.shape[0]), dtype=_out_dtype(precision))


@torch.library.custom_op("bnb_b200::policy_tail", mutates_args=(), device_types="cuda")
def policy_tail(x: Tensor, alive: Optional[Tensor], team_id: Optional[Tensor], uniforms: Tensor, heads: List[Tensor],
                pma: List[Tensor], win_cols: List[int], n_ships: int) -> Tuple[Tensor, Tensor, Tensor, Tensor]:
    """Everything of the rollout step behind the trunk under the bfloat16 contract, in six launches: the
    heads, TeamPMA, the win head on one row per team, the action draw.  x (B, N+M, 128) bfloat16 trunk
    output, uniforms (B * N, 3) float32; ``heads`` five parameters each of the action, next-state and
    value head and, with ``pma`` = [seeds, in_proj, out_proj, norm], the win head, whose outputs go to the
    columns ``win_cols`` of the value; alive (B, N+M) and team_id (B, N or more columns) are only read
    then.  Returns (action (B, N, 3) int64, logprob (B, N), value (B, N, K), pred_next (B, N, P)),
    bfloat16 but for the action."""
    return _capi.host.policy_tail(x, alive, team_id, uniforms, heads, pma, win_cols, n_ships)


@policy_tail.register_fake
def _(x, alive, team_id, uniforms, heads, pma, win_cols, n_ships):
    B = x.shape[0]
    return (x.new_empty((B, n_ships, 3), dtype=torch.int64), x.new_empty((B, n_ships)),
            x.new_empty((B, n_ships, heads[13].shape[0])), x.new_empty((B, n_ships, heads[8].shape[0])))


@torch.library.custom_op("bnb_b200::team_pma", mutates_args=(), device_types="cuda")
def team_pma(x: Tensor, team_id: Tensor, alive: Tensor, seeds: Tensor, in_proj: Tensor, out_proj: Tensor, norm_w: Tensor,
             n_heads: int, precision: int) -> Tensor:
    """``bnb_team_pma_fwd``: x (B, N, D), team_id (B, N) int, alive (B, N) bool -> (B, N, D) in x's
    dtype when that is bfloat16, else float32."""
    dev = x.device
    B, N, D = x.shape
    _check_params(dev, "TeamPMA", seeds, in_proj, out_proj, norm_w)
    with torch.cuda.device(dev):
        xin = _capi.f32c(x)
        tid = team_id.to(torch.int32).contiguous()
        al = _capi.u8(alive)
        y = torch.empty(B, N, D, device=dev, dtype=torch.bfloat16 if x.dtype == torch.bfloat16 else torch.float32)
        nbytes = _capi.lib.bnb_team_pma_scratch_bytes(D, B, N)
        scratch = torch.empty(max(int(nbytes), 256), dtype=torch.uint8, device=dev)
        st = _capi.lib.bnb_team_pma_fwd(seeds.data_ptr(), in_proj.data_ptr(), out_proj.data_ptr(), norm_w.data_ptr(), D, n_heads,
                                        xin.data_ptr(), tid.data_ptr(), al.data_ptr(), y.data_ptr(),
                                        1 if y.dtype == torch.bfloat16 else 0, B, N, precision, scratch.data_ptr(),
                                        scratch.numel(), _capi.stream_handle(dev))
    _capi.check("bnb_team_pma_fwd", st)
    return y


@team_pma.register_fake
def _(x, team_id, alive, seeds, in_proj, out_proj, norm_w, n_heads, precision):
    return x.new_empty(x.shape, dtype=torch.bfloat16 if x.dtype == torch.bfloat16 else torch.float32)


@torch.library.custom_op("bnb_b200::action_dist", mutates_args=(), device_types="cuda")
def action_dist(logits: Tensor, uniforms: Optional[Tensor], given: Optional[Tensor], want_entropy: bool) -> Tuple[Tensor, Tensor, Tensor]:
    """``bnb_action_dist_fwd`` over logits (R, 12): with ``uniforms`` (R, 3) draws an action per row
    by inverse CDF, with ``given`` (R, 3) int64 scores those actions.  Returns (action (R, 3) int64,
    logprob (R,), entropy (R,)), all float32 but the action; the action is empty when ``given`` was
    passed, the entropy is empty unless asked for."""
    dev = logits.device
    precision = _capi.BNB_BF16 if logits.dtype == torch.bfloat16 else _capi.BNB_FP32
    with torch.cuda.device(dev):
        flat = _capi.f32c(logits)
        R = flat.shape[0]
        logprob = torch.empty(R, device=dev, dtype=torch.float32)
        entropy = torch.empty(R if want_entropy else 0, device=dev, dtype=torch.float32)
        action = torch.empty(R if given is None else 0, 3, device=dev, dtype=torch.int64)
        g = None if given is None else given.to(torch.int64).contiguous()
        u = None if uniforms is None else _capi.f32c(uniforms)
        st = _capi.lib.bnb_action_dist_fwd(flat.data_ptr(), _capi.ptr(u), _capi.ptr(g), action.data_ptr() if given is None else None,
                                           logprob.data_ptr(), entropy.data_ptr() if want_entropy else None, R, precision,
                                           _capi.stream_handle(dev))
    _capi.check("bnb_action_dist_fwd", st)
    return action, logprob, entropy


@action_dist.register_fake
def _(logits, uniforms, given, want_entropy):
    R = logits.shape[0]
    return (logits.new_empty((R if given is None else 0, 3), dtype=torch.int64), logits.new_empty((R,), dtype=torch.float32),
            logits.new_empty((R if want_entropy else 0,), dtype=torch.float32))
