"""The native end of a rollout step (``bnb_b200::policy_tail``: heads, team pooling, win head, action
draw) and the encoder that skips idle bullet slots, against the same policy assembled from its modules
(which the fixtures of the reference pin) and a plain float32 pooling.
"""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


class _Obs(dict):
    bullets = None


class _Coordinator:
    total_prediction_dimension = 10

    def __init__(self, width, read):
        self.total_input_dimension = width
        self.get_input_vector = read


def _policy(N, seed=0, ks=(0, 1)):
    import boost_and_broadside_b200 as bnb
    from boost_and_broadside_b200 import workloads

    torch.manual_seed(seed)
    p = bnb.YemongPolicy(workloads.rl_config(), _Coordinator(66, lambda o: o["raw"]), 11, N, ks,
                         bullet_coordinator=_Coordinator(26, lambda o: o.bullets["raw"])).to(DEV).eval()
    with torch.no_grad():
        if ks:
            p.team_pma.seeds.normal_(0.0, 0.5)
    return p


def _obs(B, N, M, NB, seed, int_type=torch.int64):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    alive = torch.rand(B, N + M, device=DEV, generator=gen) < 0.7
    obs = _Obs(alive=alive, raw=torch.randn(B, N + M, 66, device=DEV, generator=gen),
               team_id=torch.randint(0, 2, (B, N + M), device=DEV, generator=gen).to(int_type))
    obs["alive"][0, :N] = False            # a team (here both) without a ship alive
    if NB:
        mask = torch.rand(B, NB, device=DEV, generator=gen) < 0.3
        mask[B // 2] = False
        obs.bullets = {"raw": torch.randn(B, NB, 26, device=DEV, generator=gen), "ACTIVE": mask}
    hidden = torch.randn(2, B * N, 512, device=DEV, generator=gen) * 0.5
    return obs, hidden


def _modules_step(p, obs, hidden, generator):
    """The same step through the modules one by one, every bullet slot encoded."""
    from boost_and_broadside_b200 import sample_action

    N = p._num_ships
    bullets = mask = None
    if obs.bullets is not None:
        bullets, mask = p.bullet_encoder(obs), obs.bullets["ACTIVE"]
    x, nh = p.step(p.encoder(obs), obs["alive"], hidden, bullets=bullets, bullet_mask=mask)
    xs = x[:, :N].contiguous()
    logits, pred, value = p.action_head(xs), p.next_state_head(xs), p.value_head_local(xs)
    if p._team_pma_k:
        win = p.value_head_win(p.team_pma(xs, obs["team_id"][:, :N], obs["alive"][:, :N]))
        for i, k in enumerate(p._team_pma_k):
            value[:, :, k] = win[:, :, i]
    action, logprob = sample_action(logits, generator)
    return action, logprob, value, pred, nh


@pytest.mark.parametrize("B,N,M,NB,ks", [(1, 1, 0, 0, (0, 1)), (17, 8, 4, 80, (0, 1)), (150, 3, 1, 7, (4,)), (5, 152, 0, 0, (2, 0, 10)),
                                         (40, 8, 4, 129, ()), (2500, 2, 0, 1, (0, 1))])
def test_native_tail_matches_the_modules(B, N, M, NB, ks):
    p = _policy(N, seed=B, ks=ks)
    obs, hidden = _obs(B, N, M, NB, seed=B + N, int_type=torch.int64 if B % 2 else torch.int32)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        got = p.get_action_and_value(obs, hidden, generator=torch.Generator(device=DEV).manual_seed(3))
        ref = _modules_step(p, obs, hidden, torch.Generator(device=DEV).manual_seed(3))
    for name, g, r in zip(("action", "logprob", "value", "pred_next", "hidden"), got, ref):
        assert g.shape == r.shape and g.dtype == r.dtype, name
        if name != "value":   # the same kernels' arithmetic: the same bits
            assert torch.equal(g, r), name
    err = (got[2].float() - ref[2].float()).abs().max() / ref[2].float().abs().max()
    assert float(err) <= 1e-2   # the pooled rows are projected after pooling, not before


def test_native_tail_under_torch_compile_is_one_graph_and_matches_eager():
    p = _policy(8, seed=5)
    obs, hidden = _obs(16, 8, 4, 24, seed=6)
    compiled = torch.compile(p.get_action_and_value, mode="reduce-overhead", fullgraph=True)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        _, _, v0, p0, h0 = p.get_action_and_value(obs, hidden)
        for _ in range(3):
            _, _, v, pn, h = compiled(obs, hidden)
            v, pn, h = v.clone(), pn.clone(), h.clone()
    assert torch.equal(v, v0) and torch.equal(pn, p0) and torch.equal(h, h0)


def test_value_columns_count_from_the_end_as_indexing_does():
    p = _policy(4, seed=2, ks=(-1, -11, 3))
    obs, hidden = _obs(9, 4, 1, 0, seed=8)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        got = p.get_action_and_value(obs, hidden, generator=torch.Generator(device=DEV).manual_seed(3))
        ref = _modules_step(p, obs, hidden, torch.Generator(device=DEV).manual_seed(3))
        assert float((got[2].float() - ref[2].float()).abs().max()) <= 1e-2 * float(ref[2].float().abs().max())
        p._team_pma_k = (11,)
        with pytest.raises(IndexError):
            p.get_action_and_value(obs, hidden)


def test_without_a_team_value_neither_teams_nor_alive_flags_are_needed():
    p = _policy(4, seed=2, ks=())
    obs, hidden = _obs(9, 4, 1, 0, seed=8)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        full = p.get_action_and_value(obs, hidden, generator=torch.Generator(device=DEV).manual_seed(3))
        del obs["team_id"]
        bare = p.get_action_and_value(obs, hidden, generator=torch.Generator(device=DEV).manual_seed(3))
        assert all(torch.equal(a, b) for a, b in zip(full, bare))
        obs["alive"] = None
        p.get_action_and_value(obs, hidden)


def test_a_short_team_id_raises():
    p = _policy(4, seed=2)
    obs, hidden = _obs(9, 4, 1, 0, seed=8)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        whole = p.get_action_and_value(obs, hidden, generator=torch.Generator(device=DEV).manual_seed(3))
        team = obs["team_id"]
        obs["team_id"] = team[:, :4]   # the ships' columns are enough, at any stride
        ships = p.get_action_and_value(obs, hidden, generator=torch.Generator(device=DEV).manual_seed(3))
        assert all(torch.equal(a, b) for a, b in zip(whole, ships))
        for short in (team[:, :3], team[:8]):
            obs["team_id"] = short
            with pytest.raises(RuntimeError, match="team_id"):
                p.get_action_and_value(obs, hidden)


def test_replaced_heads_and_hooks_are_called():
    import boost_and_broadside_b200 as bnb

    p = _policy(4, seed=2)
    obs, hidden = _obs(9, 4, 1, 6, seed=8)
    seen = []
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        for module in (p.action_head, p.team_pma, p.next_state_head, p.bullet_encoder):
            handle = module.register_forward_hook(lambda m, a, out: seen.append(m))
            got = p.get_action_and_value(obs, hidden, generator=torch.Generator(device=DEV).manual_seed(3))
            handle.remove()
            assert seen[-1] is module

        class Doubled(bnb.HeadMLP):
            def forward(self, x):
                return 2 * super().forward(x)

        doubled = Doubled(128, 10).to(DEV)
        doubled.load_state_dict(p.next_state_head.net.state_dict())
        p.next_state_head.net = doubled
        twice = p.get_action_and_value(obs, hidden, generator=torch.Generator(device=DEV).manual_seed(3))
        assert torch.equal(twice[3], 2 * got[3])


def _move_off_16_bytes(module, name):
    p = getattr(module, name)
    flat = torch.empty(p.numel() + 1, device=DEV)
    view = flat[1:].view(p.shape).copy_(p.detach())
    assert view.data_ptr() % 16 == 4
    p.data = view


def test_parameters_that_start_between_16_byte_boundaries():
    """Copied where any start was taken before (biases, gains, seeds, a head's second weight, first weights of
    odd widths), refused where it was refused."""
    p = _policy(6, seed=4)
    obs, hidden = _obs(21, 6, 2, 9, seed=9)
    step = lambda: p.get_action_and_value(obs, hidden, generator=torch.Generator(device=DEV).manual_seed(3))
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        ref = step()
        _move_off_16_bytes(p.team_pma, "seeds")
        _move_off_16_bytes(p.team_pma.norm, "weight")
        for head in (p.action_head, p.value_head_local, p.value_head_win, p.next_state_head.net):
            for module, name in ((head[0], "bias"), (head[1], "weight"), (head[3], "weight"), (head[3], "bias")):
                _move_off_16_bytes(module, name)
        for chain in (p.encoder.feature_extractor, p.bullet_encoder.net):   # 66 and 26 columns
            for module, name in ((chain[0], "weight"), (chain[0], "bias"), (chain[1], "weight"), (chain[3], "bias"), (chain[4], "weight")):
                _move_off_16_bytes(module, name)
        for a, b in zip(step(), ref):
            assert torch.equal(a, b)
        for module, name in ((p.action_head[0], "weight"), (p.team_pma.attn, "in_proj_weight"), (p.team_pma.attn.out_proj, "weight"),
                             (p.encoder.feature_extractor[3], "weight")):
            held = getattr(module, name).data
            _move_off_16_bytes(module, name)
            with pytest.raises(RuntimeError, match="align"):
                step()
            getattr(module, name).data = held
        for a, b in zip(step(), ref):
            assert torch.equal(a, b)


def test_parameters_that_are_transposed_views():
    """An encoder's first weight and a head's second one (and its bias) are copied when they are strided."""
    p = _policy(6, seed=4)
    obs, hidden = _obs(21, 6, 2, 9, seed=9)
    step = lambda: p.get_action_and_value(obs, hidden, generator=torch.Generator(device=DEV).manual_seed(3))
    heads = (p.action_head, p.value_head_local, p.value_head_win, p.next_state_head.net)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        ref, x = step(), torch.randn(70, 128, device=DEV).to(torch.bfloat16)
        rows = [h(x) for h in heads]
        for linear in (p.encoder.feature_extractor[0], p.bullet_encoder.net[0], *(h[3] for h in heads)):
            linear.weight.data = linear.weight.data.t().contiguous().t()
            assert not linear.weight.is_contiguous()
        for h in heads:
            h[3].bias.data = torch.stack([h[3].bias.data, h[3].bias.data], dim=1)[:, 0]
        for a, b in zip([*step(), *(h(x) for h in heads)], [*ref, *rows]):
            assert torch.equal(a, b)
        p.action_head[0].weight.data = p.action_head[0].weight.data.t().contiguous().t()
        with pytest.raises(RuntimeError, match="contiguous"):
            step()
    with torch.no_grad():   # float32: a first weight of whole 32-column pieces goes in without a padded copy
        from boost_and_broadside_b200 import _capi
        ps = [torch.randn(256, 64, device=DEV), *(torch.randn(256, device=DEV) for _ in range(2)), torch.randn(128, 256, device=DEV),
              *(torch.randn(128, device=DEV) for _ in range(2))]
        raw = torch.randn(33, 64, device=DEV)
        a = _capi.host.mlp_chain(raw, ps, _capi.BNB_FP32, None)
        b = _capi.host.mlp_chain(raw, [ps[0].t().contiguous().t(), *ps[1:]], _capi.BNB_FP32, None)
        assert torch.equal(a, b)


def test_a_policy_without_a_team_value_compiles_to_one_graph():
    p = _policy(8, seed=5, ks=())
    obs, hidden = _obs(16, 8, 4, 24, seed=6)
    compiled = torch.compile(p.get_action_and_value, mode="reduce-overhead", fullgraph=True)
    with torch.no_grad(), torch.autocast(DEV, dtype=torch.bfloat16):
        _, _, v0, p0, h0 = p.get_action_and_value(obs, hidden)
        for _ in range(3):
            _, _, v, pn, h = compiled(obs, hidden)
            v, pn, h = v.clone(), pn.clone(), h.clone()
    assert torch.equal(v, v0) and torch.equal(pn, p0) and torch.equal(h, h0)
