"""Opaque ``torch.library`` operators around the C ABI.

``torch.compile(policy)`` (the reference trains and evaluates through it,
train/rl/ppo.py:396-400) must neither trace into ctypes nor break CUDA-graph capture, so the
calls into the library are registered as custom operators: Dynamo sees one opaque node with a
shape-only fake implementation.  The real implementations are native code (csrc/host_path.cpp),
which eager calls that nobody has to see (``direct``) enter without the operator dispatcher; the
single-sublayer operator builds its ctypes structs here.  Nothing here synchronises.

``trunk_forward`` carries an autograd formula (``trunk_backward`` -> ``bnb_trunk_sequence_bwd``,
environments of one size, recomputing activations); a call known to need gradients goes through
``trunk_forward_train`` instead, which keeps its activations for the backward.  Either way a step or
sequence through ``YemongBlock`` / ``YemongTrunk`` can be differentiated with respect to tokens,
recurrent state, bullet tokens and parameters.  The
single-sublayer operators are forward-only and their module methods refuse inputs that require grad.
"""

from __future__ import annotations

import os
from typing import List, Optional, Tuple

import torch
from torch import Tensor
from torch.autograd import forward_ad

from .. import _capi
from ._weights import N_SPATIAL, packed_image, spatial_struct_from

# geom: the integers of a call, in this order
(G_BLOCKS, G_SPATIAL, G_TEMPORAL, G_HEADS, G_BULLET_CROSS, G_FIELD_SUB, G_ENVS, G_TOKENS_PER_ENV, G_SHIPS_PER_ENV,
 G_MAX_TOKENS, G_TOTAL_TOKENS, G_TOTAL_SHIPS, G_TILES, G_TIMESTEPS, G_ENGINE, G_PRECISION) = range(16)


def _debug_check(fn: str, dev: torch.device, precision: int) -> None:
    """With BNB_DEBUG_SYNC=1 in the environment every call waits for its kernels and raises if
    one of the tensor-core kernels' bounded waits ran out (status word at the head of the scratch
    buffer).  Off by default: the check synchronises, so it cannot run under graph capture."""
    if precision == _capi.BNB_BF16 and os.environ.get("BNB_DEBUG_SYNC") == "1" and not torch.cuda.is_current_stream_capturing():
        st = _capi.tensor_engine_status(dev)
        if 100 < st < 200:   # the ST_TIMEOUT_* codes; other values are scratch data of the exact engine
            raise RuntimeError(f"{fn}: a bounded wait of the tensor-core kernels ran out (code {st})")


def _raise_pending_status(dev: torch.device) -> None:
    """A bounded wait of an earlier call on this device ran out (its kernels drained and its
    outputs were garbage): say so once, at the next call, without synchronising."""
    with torch.cuda.device(dev):
        st = _capi.lib.bnb_last_status()
        if st:
            _capi.lib.bnb_clear_status()
            raise RuntimeError(
                f"an earlier tensor-core call on {dev} gave up a bounded wait: {_capi.lib.bnb_status_string(st).decode()} "
                f"(status {st}); its outputs, and any state carried from them, are invalid")


_dispatch_modes, _function_transform, _jit_trace = (torch._C._len_torch_dispatch_stack, torch._C._functorch.peek_interpreter_stack,
                                                    torch._C._get_tracing_state)


def direct(t: Tensor) -> bool:
    """Whether an operator's body may be called as it is: an ordinary eager tensor, and nobody at work who has
    to see the operator: a compiler, TorchScript's tracer, a dispatch mode (make_fx, flop counting), a
    function transform (vmap) or forward-mode differentiation, whose tangents the body would drop."""
    return (not torch.compiler.is_compiling() and type(t) is Tensor and not _dispatch_modes() and _function_transform() is None
            and _jit_trace() is None and forward_ad._current_level < 0)


def uniform_geom(n_envs: int, tokens: int, ships: int) -> List[int]:
    """Batch part of ``geom`` for environments of one size (entries G_ENVS .. G_TILES)."""
    return [n_envs, tokens, ships, tokens, n_envs * tokens, n_envs * ships, 0]


def _batch(geom: List[int], offsets: List[Tensor]) -> "_capi.Batch":
    if offsets:
        tok, ship = offsets[0], offsets[1]
        tiles = offsets[2] if len(offsets) > 2 else None
        ids = offsets[3] if len(offsets) > 3 else None
        return _capi.Batch(geom[G_ENVS], 0, 0, geom[G_MAX_TOKENS], geom[G_TOTAL_TOKENS], geom[G_TOTAL_SHIPS],
                           tok.data_ptr(), ship.data_ptr(), _capi.ptr(tiles), _capi.ptr(ids), geom[G_TILES])
    return _capi.Batch(geom[G_ENVS], geom[G_TOKENS_PER_ENV], geom[G_SHIPS_PER_ENV], geom[G_MAX_TOKENS],
                       geom[G_TOTAL_TOKENS], geom[G_TOTAL_SHIPS], None, None, None, None, 0)


@torch.library.custom_op("bnb_b200::trunk_forward", mutates_args=(), device_types="cuda")
def trunk_forward(
    x: Tensor,
    alive: Optional[Tensor],
    hidden: Tensor,
    done: Optional[Tensor],
    reset_env: Optional[Tensor],
    bullets: Optional[Tensor],
    bullet_mask: Optional[Tensor],
    weights: List[Tensor],
    offsets: List[Tensor],
    geom: List[int],
) -> Tuple[Tensor, Tensor]:
    """Blocks of (spatial sublayers, temporal sublayers) over x: ``bnb_trunk_step`` when
    geom[G_TIMESTEPS] is 0, else ``bnb_trunk_sequence`` over that many timesteps.

    x (total_tokens, D) or (T, total_tokens, D), float32 or bfloat16; hidden (L, total_ships, 4D) packed;
    ``weights`` the parameters of every sublayer, block-major, spatial before temporal inside a
    block, each sublayer in the order of ``_weights.spatial_tensors`` / ``temporal_tensors``;
    ``offsets`` empty for environments of one size, else [tok_off, ship_off(, tile_env_begin,
    tile_env_ids)].  Returns (y like x: bfloat16 for bfloat16 tokens, else float32; new hidden like
    hidden, float32).
    """
    return trunk_call(x, alive, hidden, done, reset_env, bullets, bullet_mask, weights, offsets, geom)


def trunk_call(x, alive, hidden, done, reset_env, bullets, bullet_mask, weights, offsets, geom):
    """The body of ``trunk_forward``, in native code (csrc/host_path.cpp); eager calls without gradients
    come here directly, past the operator dispatcher."""
    out = _capi.host.trunk_forward(x, alive, hidden, done, reset_env, bullets, bullet_mask, weights, offsets, geom, _capi.scratch_for)
    if geom[G_PRECISION] == _capi.BNB_BF16:
        fn = "bnb_trunk_step" if geom[G_TIMESTEPS] == 0 else "bnb_trunk_sequence"
        _capi.note_engine_choice(fn)
        _debug_check(fn, x.device, geom[G_PRECISION])
    return out


@trunk_forward.register_fake
def _trunk_forward_fake(x, alive, hidden, done, reset_env, bullets, bullet_mask, weights, offsets, geom):
    out_dtype = torch.bfloat16 if x.dtype == torch.bfloat16 else torch.float32
    return (x.new_empty(x.shape, dtype=out_dtype), hidden.new_empty(hidden.shape, dtype=torch.float32))


def _grad_precision(geom: List[int]) -> int:
    """Precision of the training forward and the backward: bf16 operands after an autocast forward."""
    return _capi.BNB_BF16 if geom[G_PRECISION] == _capi.BNB_BF16 else _capi.BNB_FP32


def _kept_size(geom: List[int], d_model: int, bullets_per_env: int) -> int:
    """Bytes of the kept-activation buffer of a training forward (host arithmetic only)."""
    need = _capi.lib.bnb_trunk_kept_bytes(geom[G_BLOCKS], geom[G_SPATIAL], geom[G_TEMPORAL], d_model, geom[G_HEADS],
                                          _batch(geom, []), max(1, geom[G_TIMESTEPS]), bullets_per_env, _grad_precision(geom))
    return max(256, int(need))


@torch.library.custom_op("bnb_b200::trunk_backward", mutates_args=(), device_types="cuda")
def trunk_backward(
    dy: Tensor,
    dhidden_out: Optional[Tensor],
    kept: Optional[Tensor],
    x: Tensor,
    alive: Optional[Tensor],
    hidden: Tensor,
    done: Optional[Tensor],
    bullets: Optional[Tensor],
    bullet_mask: Optional[Tensor],
    weights: List[Tensor],
    geom: List[int],
) -> List[Tensor]:
    """Gradients of ``trunk_forward`` (environments of one size, no ``reset_env``) through
    ``bnb_trunk_sequence_bwd``: float32 tensors throughout; after a forward under bf16 autocast the
    Linear products round their operands to bfloat16, as the reference's backward does there.  Returns
    [d x, d hidden, d bullets (empty without bullets), every parameter gradient in one flat buffer
    (``_split_grads`` cuts it into one view per tensor of ``weights``)].
    ``kept``: the activations ``trunk_forward_train`` kept for this call (the backward consumes
    them), or None: every sublayer's intermediates are recomputed."""
    return _capi.host.trunk_backward(dy, dhidden_out, kept, x, alive, hidden, done, bullets, bullet_mask, weights, geom)


@trunk_backward.register_fake
def _trunk_backward_fake(dy, dhidden_out, kept, x, alive, hidden, done, bullets, bullet_mask, weights, geom):
    dbul = x.new_empty(bullets.shape, dtype=torch.float32) if bullets is not None and geom[G_BULLET_CROSS] > 0 else x.new_empty(0, dtype=torch.float32)
    return [x.new_empty(x.shape, dtype=torch.float32), hidden.new_empty(hidden.shape, dtype=torch.float32), dbul,
            x.new_empty(sum(_grad_sizes(weights)), dtype=torch.float32)]


def _grad_sizes(weights: List[Tensor]) -> List[int]:
    """Elements each parameter gradient takes in the flat buffer (16-byte granules)."""
    return [(w.numel() + 3) // 4 * 4 for w in weights]


def _split_grads(flat: Tensor, weights: List[Tensor]) -> List[Tensor]:
    views, off = [], 0
    for w, n in zip(weights, _grad_sizes(weights)):
        views.append(flat[off : off + w.numel()].view(w.shape))
        off += n
    return views


def _shape_grads(out, x, hidden, bullets, weights):
    dx, dh, dbul, dws = out[0], out[1], out[2], _split_grads(out[3], weights)
    dx = dx.reshape(x.shape).to(x.dtype)
    dh = dh.reshape(hidden.shape).to(hidden.dtype)
    dbul = dbul.reshape(bullets.shape).to(bullets.dtype) if bullets is not None and dbul.numel() else None
    return dx, dh, dbul, [g.to(w.dtype) for g, w in zip(dws, weights)]


def _trunk_setup_context(ctx, inputs, output):
    x, alive, hidden, done, reset_env, bullets, bullet_mask, weights, offsets, geom = inputs
    ctx.geom = list(geom)
    ctx.unsupported = ("a ragged batch" if offsets else "reset_env" if reset_env is not None else "")
    ctx.n_offsets = len(offsets)
    ctx.save_for_backward(x, alive, hidden, done, bullets, bullet_mask, *weights)


def _trunk_backward_formula(ctx, dy, dhidden_out):
    if ctx.unsupported:
        raise NotImplementedError(f"the CUDA trunk's backward does not cover {ctx.unsupported}; run that call under torch.no_grad()")
    x, alive, hidden, done, bullets, bullet_mask, *weights = ctx.saved_tensors
    out = trunk_backward(dy, dhidden_out, None, x, alive, hidden, done, bullets, bullet_mask, list(weights), ctx.geom)
    dx, dh, dbul, dws = _shape_grads(out, x, hidden, bullets, weights)
    # one entry per input; a list input takes a list of the same length
    return dx, None, dh, None, None, dbul, None, dws, [None] * ctx.n_offsets, None


trunk_forward.register_autograd(_trunk_backward_formula, setup_context=_trunk_setup_context)


@torch.library.custom_op("bnb_b200::trunk_forward_train", mutates_args=(), device_types="cuda")
def trunk_forward_train(
    x: Tensor,
    alive: Optional[Tensor],
    hidden: Tensor,
    done: Optional[Tensor],
    bullets: Optional[Tensor],
    bullet_mask: Optional[Tensor],
    weights: List[Tensor],
    geom: List[int],
) -> Tuple[Tensor, Tensor, Tensor]:
    """``trunk_forward`` for a call that will be differentiated (environments of one size, no
    ``reset_env``): ``bnb_trunk_sequence_fwd_train`` runs the trunk sublayer by sublayer and keeps
    every sublayer's intermediates, as autograd does for the reference without grad_checkpoint;
    the backward then skips its recomputation.  Returns (y, new hidden, kept activations); y is
    float32, or bfloat16 for bfloat16 tokens."""
    return _capi.host.trunk_forward_train(x, alive, hidden, done, bullets, bullet_mask, weights, geom)


@trunk_forward_train.register_fake
def _trunk_forward_train_fake(x, alive, hidden, done, bullets, bullet_mask, weights, geom):
    out_dtype = torch.bfloat16 if x.dtype == torch.bfloat16 else torch.float32
    per_env = bullets.shape[1] if bullets is not None and geom[G_BULLET_CROSS] > 0 else 0
    return (x.new_empty(x.shape, dtype=out_dtype), hidden.new_empty(hidden.shape, dtype=torch.float32),
            x.new_empty(_kept_size(geom, x.shape[-1], per_env), dtype=torch.uint8))


def _train_setup_context(ctx, inputs, output):
    x, alive, hidden, done, bullets, bullet_mask, weights, geom = inputs
    ctx.geom = list(geom)
    ctx.consumed = False
    ctx.mark_non_differentiable(output[2])
    # autograd would otherwise materialise a zero "gradient" the size of the kept activations
    ctx.set_materialize_grads(False)
    ctx.save_for_backward(x, alive, hidden, done, bullets, bullet_mask, output[2], *weights)


def _train_backward_formula(ctx, dy, dhidden_out, _dkept):
    if ctx.consumed:
        raise RuntimeError("the kept activations of this trunk call were consumed by an earlier backward; for a second "
                           "backward through the same graph set BNB_GRAD_MODE=recompute")
    ctx.consumed = True
    x, alive, hidden, done, bullets, bullet_mask, kept, *weights = ctx.saved_tensors
    if dy is None:
        dy = torch.zeros_like(x, dtype=torch.float32)
    out = trunk_backward(dy, dhidden_out, kept, x, alive, hidden, done, bullets, bullet_mask, list(weights), ctx.geom)
    dx, dh, dbul, dws = _shape_grads(out, x, hidden, bullets, weights)
    return dx, None, dh, None, dbul, None, dws, None


trunk_forward_train.register_autograd(_train_backward_formula, setup_context=_train_setup_context)


@torch.library.custom_op("bnb_b200::spatial_forward", mutates_args=(), device_types="cuda")
def spatial_forward(
    x: Tensor,
    alive: Optional[Tensor],
    bullets: Optional[Tensor],
    bullet_mask: Optional[Tensor],
    weights: List[Tensor],
    n_heads: int,
    precision: int,
    engine: int,
) -> Tensor:
    """One spatial sublayer, ``bnb_spatial_block_fwd``: x (B, N, D), alive (B, N) or None,
    bullets (B, NB, D) / bullet_mask (B, NB) or None; returns float32 (B, N, D)."""
    dev = x.device
    B, N, D = x.shape
    ts = list(weights)
    with torch.cuda.device(dev):
        xin = _capi.f32c(x)
        alive_u8 = _capi.u8(alive)
        y = torch.empty_like(xin)
        batch = _capi.uniform_batch(B, N, N)
        bul = _capi.BulletArgs(bullets if len(ts) > N_SPATIAL else None, bullet_mask, B, D)
        nbytes = _capi.lib.bnb_scratch_bytes(D, batch, 1, bul.per_env)
        scratch = _capi.scratch_for(dev, nbytes)
        _raise_pending_status(dev)
        w = spatial_struct_from(ts, dev, packed_image("spatial", ts, n_heads, dev, precision, engine))
        st = _capi.lib.bnb_spatial_block_fwd(
            w, D, n_heads, xin.data_ptr(), _capi.ptr(alive_u8), bul.arg, y.data_ptr(), batch, 1, precision, engine,
            scratch.data_ptr(), scratch.numel(), _capi.stream_handle(dev),
        )
    _capi.check("bnb_spatial_block_fwd", st)
    _capi.note_engine_choice("bnb_spatial_block_fwd")
    _debug_check("bnb_spatial_block_fwd", dev, precision)
    return y


@spatial_forward.register_fake
def _spatial_forward_fake(x, alive, bullets, bullet_mask, weights, n_heads, precision, engine):
    return x.new_empty(x.shape, dtype=torch.float32)
