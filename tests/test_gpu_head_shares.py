"""The four heads of the native tail in one launch: row tiles of the ships' three chains and of the teams' one shared out over the
CTAs, from one tile each to several rounds, more team rows than ships among them, against the modules one by one (the same
arithmetic per row: the same bits)."""

import pytest
import torch

from tests.test_gpu_policy_tail import _modules_step, _obs, _policy

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,N", [(1, 1), (64, 1), (65, 2), (4736, 1), (4737, 1), (9500, 1), (1579, 12), (2400, 8)])
def test_heads_and_win_head(B, N):
    p = _policy(N, seed=B + N)
    obs, hidden = _obs(B, N, 1, 0, B)
    run = lambda f: f(torch.Generator(device=DEV).manual_seed(3))  # noqa: E731
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        native = run(lambda g: p.get_action_and_value(obs, hidden, g))
        modules = run(lambda g: _modules_step(p, obs, hidden, g))
    for name, a, b in zip(("value", "next state", "hidden"), native[2:], modules[2:]):
        if name == "value":   # the win columns come through another order of pooling and projection: the other test's bound
            assert torch.equal(a[..., 2:], b[..., 2:]), name
            assert float((a.float() - b.float()).abs().max()) <= 1e-2 * float(b.float().abs().max()), name
        else:
            assert torch.equal(a, b), name
