"""Scratch of a differentiated call by its bullet slots (host arithmetic of the library; no GPU)."""

import pytest

from boost_and_broadside_b200 import _capi


@pytest.mark.parametrize("precision", ["BNB_BF16", "BNB_FP32"])
@pytest.mark.parametrize("envs,steps,tokens,slots", [(1, 1, 1, 1), (96, 16, 12, 80), (7, 3, 40, 33), (1024, 32, 8, 5)])
def test_scratch_of_bullet_slots(envs, steps, tokens, slots, precision):
    """Per slot the normed row (128 floats) and its root, keys and values (256), their gradient (256) and that of the token (128); the list
    and the rows of the slots in use stand in these.  Five areas, each rounded up to 256 bytes."""
    batch = _capi.uniform_batch(envs, tokens, tokens)
    need = lambda nb: _capi.lib.bnb_trunk_bwd_scratch_bytes(2, 2, 1, 128, batch, steps, nb, getattr(_capi, precision))  # noqa: E731
    assert need(slots) - need(0) <= 4 * (6 * 128 + 1) * steps * envs * slots + 5 * 256
