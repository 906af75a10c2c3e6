"""What the native end of the policy step refuses before anything is launched: on CPU tensors, whose device
is the last thing it looks at."""

from __future__ import annotations

import pytest
import torch

B, N, M, D = 3, 5, 2, 128


def _head(out):
    return [torch.zeros(2 * D, D), torch.zeros(2 * D), torch.ones(2 * D), torch.zeros(out, 2 * D), torch.zeros(out)]


def _call(**change):
    from boost_and_broadside_b200 import _capi

    a = dict(x=torch.zeros(B, N + M, D, dtype=torch.bfloat16), alive=torch.ones(B, N + M, dtype=torch.bool),
             team_id=torch.zeros(B, N + M, dtype=torch.int64), uniforms=torch.zeros(B * N, 3),
             heads=[*_head(12), *_head(10), *_head(11), *_head(2)],
             pma=[torch.zeros(2, D), torch.zeros(3 * D, D), torch.zeros(D, D), torch.ones(D)], win_cols=[0, 1], n_ships=N)
    a.update(change)
    return _capi.host.policy_tail(a["x"], a["alive"], a["team_id"], a["uniforms"], a["heads"], a["pma"], a["win_cols"], a["n_ships"])


@pytest.mark.parametrize("cols", [[11], [0, 11], [-12], [256], [1 << 40]])
def test_value_columns_outside_the_value_raise(cols):
    with pytest.raises(IndexError, match="out of bounds"):
        _call(win_cols=cols)


def test_more_value_columns_than_the_win_head_has_raise():
    with pytest.raises(IndexError, match="out of bounds"):
        _call(win_cols=[0, 1, 2])


def test_inputs_in_order_reach_the_device_check():
    for cols in ([0, 1], [-1], [10, -11]):
        with pytest.raises(RuntimeError, match="(?i)cuda"):
            _call(win_cols=cols)


@pytest.mark.parametrize("change", [
    dict(team_id=torch.zeros(B, N - 1, dtype=torch.int64)), dict(team_id=torch.zeros(B - 1, N + M, dtype=torch.int64)),
    dict(team_id=torch.zeros(N + M, dtype=torch.int64)), dict(team_id=None), dict(alive=torch.ones(B, N, dtype=torch.bool)), dict(alive=None),
    dict(uniforms=torch.zeros(B * N - 1, 3)), dict(uniforms=torch.zeros(B * N, 3, dtype=torch.float64)), dict(n_ships=N + M + 1),
    dict(pma=[torch.zeros(1, D), torch.zeros(3 * D, D), torch.zeros(D, D), torch.ones(D)]),
    dict(pma=[torch.zeros(2, D), torch.zeros(2 * D, D), torch.zeros(D, D), torch.ones(D)]),
    dict(heads=[*_head(12), *_head(10), *_head(11)]), dict(heads=[*_head(12), *_head(33), *_head(11), *_head(2)]),
    dict(heads=[torch.zeros(D, D), *_head(12)[1:], *_head(10), *_head(11), *_head(2)]),
    dict(heads=[*_head(12)[:4], torch.zeros(11), *_head(10), *_head(11), *_head(2)])])
def test_inputs_of_other_sizes_raise(change):
    with pytest.raises(RuntimeError, match="must|served|expected"):
        _call(**change)


def test_team_id_of_the_ships_alone_is_enough_and_none_without_a_team_value():
    no_team = dict(heads=[*_head(12), *_head(10), *_head(11)], pma=[], win_cols=[])
    for change in (dict(team_id=torch.zeros(B, N, dtype=torch.int32)), dict(no_team, team_id=None, alive=None)):
        with pytest.raises(RuntimeError, match="(?i)cuda"):
            _call(**change)


def test_rows_wanted_of_an_encoder_are_as_many_as_its_rows():
    from boost_and_broadside_b200 import _capi

    with pytest.raises(RuntimeError, match="one element per row"):
        _capi.host.mlp_chain(torch.zeros(8, D), [*_head(12)], _capi.BNB_BF16, torch.ones(7, dtype=torch.bool))


def test_only_policies_of_the_built_sizes_take_the_native_end():
    from boost_and_broadside_b200 import _capi

    head = lambda out, hidden=256, width=128: [width, hidden, out]
    ok = _capi.host.tail_supported
    assert ok(128, 4, 8, [*head(12), *head(10), *head(11), *head(2)])
    for other in ([*head(12, 128), *head(10)], [*head(12), *head(10, 512)], [*head(12), *head(10), *head(11, 256, 64)], [*head(11), *head(10)], []):
        assert not ok(128, 4, 8, other)
