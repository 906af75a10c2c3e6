"""Rows on 16-byte but not on 32-byte boundaries take the tile kernel's narrower accesses: same bits."""

import pytest
import torch

from tests.helpers import build_trunk

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _shifted(t: torch.Tensor) -> torch.Tensor:
    """The same values 16 bytes past an aligned address."""
    step = 16 // t.element_size()
    out = torch.empty(t.numel() + step, dtype=t.dtype, device=t.device)[step:].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 32 == 16
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("what", ["x", "hidden"])
def test_narrow_rows_give_the_same_bits(dtype, what):
    g = torch.Generator(device=DEV).manual_seed(5)
    trunk = build_trunk([128, 4, 2, 2, 1, 1]).to(DEV)
    x = torch.randn(3, 23, 12, 128, device=DEV, generator=g).to(dtype)
    hidden = torch.randn(2, 23 * 8, 512, device=DEV, generator=g) * 0.5
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        for call in (lambda a, h: trunk.step(a[0], None, h), lambda a, h: trunk.sequence(a, None, h)):
            ref = call(x, hidden)
            got = call(_shifted(x) if what == "x" else x, _shifted(hidden) if what == "hidden" else hidden)
            assert all(torch.equal(a, b) for a, b in zip(got, ref))
