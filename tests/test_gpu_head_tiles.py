"""Heads and ship encoder on 128-row tiles: rows around one tile and above one tile per SM, odd and full output widths,
odd and even input widths, both input types, against the CPU oracle."""

import pytest
import torch

from oracle import trunk_oracle as O
from tests.helpers import norm_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _params(g, in_dim, out):
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    return [r(256, in_dim) / in_dim ** 0.5, 0.1 * r(256), 1 + 0.1 * r(256), r(out, 256) / 16, 0.1 * r(out)]


@pytest.mark.parametrize("rows,out,dtype", [(1, 12, torch.bfloat16), (127, 11, torch.float32), (128, 32, torch.bfloat16), (129, 1, torch.bfloat16),
                                            (148 * 128 + 5, 10, torch.bfloat16), (300 * 128, 12, torch.float32)])
def test_head_rows(rows, out, dtype):
    import boost_and_broadside_b200 as bnb

    g = torch.Generator().manual_seed(rows)
    ps = _params(g, 128, out)
    x = torch.randn(rows, 128, generator=g).to(dtype)
    head = bnb.HeadMLP(128, out)
    with torch.no_grad():
        for p, v in zip(head.parameter_list(), ps):
            p.copy_(v)
        head = head.to(DEV)
        with torch.autocast(DEV, dtype=torch.bfloat16):
            got = head(x.to(DEV))
    assert norm_err(got.float().cpu(), O.head_mlp(x.float(), *ps, "bf16").float()) < 2e-2


@pytest.mark.parametrize("rows,in_dim", [(1, 66), (127, 65), (128, 2), (129, 128), (148 * 128 + 3, 66), (300 * 128, 100)])
def test_encoder_rows(rows, in_dim):
    from boost_and_broadside_b200 import _capi
    from boost_and_broadside_b200.yemong import _end_ops

    g = torch.Generator().manual_seed(rows)
    ps = _params(g, in_dim, 128) + [1 + 0.1 * torch.randn(128, generator=g)]
    x = torch.randn(rows, in_dim, generator=g)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        got = _end_ops.mlp_call(x.to(DEV), *[p.to(DEV) for p in ps], _capi.current_precision(torch.device(DEV, 0)))
    assert norm_err(got.float().cpu(), O.encoder_mlp(x, *ps, "bf16").float()) < 2e-2
