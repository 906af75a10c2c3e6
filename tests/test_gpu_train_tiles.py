"""The training kernels of d_model 128 at the edges of their tiles: bfloat16 gradients against the float32 path
of the same call, which the oracle pins elsewhere."""

import pytest
import torch

from tests.helpers import build_trunk, norm_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


# rows T * B * (N + M): 1, 127 .. 129, above one tile per SM; tokens per environment around 8, 16 and 32; bullet slots
# around 32 and the largest ring; ship rows only, field rows only
@pytest.mark.parametrize("T,B,N,M,NB", [(1, 1, 1, 0, 0), (1, 127, 1, 0, 1), (2, 16, 3, 1, 2), (3, 43, 1, 0, 0), (9, 265, 5, 3, 0), (2, 5, 8, 0, 32),
                                        (2, 5, 9, 0, 33), (1, 3, 12, 4, 160), (2, 3, 17, 0, 80), (1, 2, 32, 0, 7), (1, 2, 33, 0, 7), (3, 4, 0, 5, 3)])
def test_bf16_gradients_near_float32(T, B, N, M, NB):
    g = torch.Generator(device=DEV).manual_seed(T * 1000 + B)
    trunk = build_trunk([128, 4, 1, 2, 1, 1]).to(DEV)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    x = r(T, B, N + M, 128).requires_grad_()
    hidden = (0.5 * r(1, B * N, 512)).requires_grad_()
    bullets = r(T * B, NB, 128).requires_grad_() if NB else None
    alive = torch.rand(T, B, N + M, device=DEV, generator=g) < 0.8
    alive[0, 0] = False
    mask = torch.rand(T * B, NB, device=DEV, generator=g) < 0.4 if NB else None
    done = torch.rand(T, B, device=DEV, generator=g) < 0.2
    dy = r(T, B, N + M, 128)
    inputs = [t for t in (x, hidden, bullets) if t is not None and t.numel()] + [p for n, p in trunk.named_parameters() if M or "field_sub" not in n]

    def grads(on):
        with torch.autocast(DEV, dtype=torch.bfloat16, enabled=on):
            y, _ = trunk.sequence(x, alive, hidden, done, bullets=bullets, bullet_mask=mask)
        return [y, *torch.autograd.grad(y.float(), inputs, dy, allow_unused=True)]

    for a, b in zip(grads(True), grads(False)):
        assert (a is None) == (b is None)
        if a is not None and float(b.abs().max()) > 0:
            assert torch.isfinite(a).all()
            assert norm_err(a.float(), b.float()) < 4e-2
