"""Which kernel a step goes to and how its work is shared out: decisions made on the host, on the CPU."""
from types import SimpleNamespace

import pytest
import torch

from cpmcu_b200.ops.dry import DryOps, dry_context
from cpmcu_b200.ops.ops import Ops


@pytest.mark.parametrize("d", [32, 64, 96, 128])
def test_counters_are_given_only_for_shares_that_the_last_block_can_add_up(d):
    """A sequence has as many shares as the caller asks for, and the block that adds them up has room for 32."""
    ops = SimpleNamespace(workspace=object(), arrivals=torch.zeros(16384, dtype=torch.int32), MAX_JOINED_SHARES=Ops.MAX_JOINED_SHARES)
    for n_splits in (2, 16, 32, 33, 64, 1000):
        got = Ops._arrivals(ops, 2, 16, 2, d, n_splits)
        assert (got is not None) == (d <= 64 and n_splits <= 32), n_splits


@pytest.mark.parametrize("n,n_heads,n_kv,d,alone", [(57, 32, 2, 128, True), (74, 32, 2, 128, True), (75, 32, 2, 128, False), (2048, 32, 2, 128, False),
                                                    (148, 16, 2, 64, True), (149, 16, 2, 64, False), (40, 80, 2, 64, True), (50, 80, 2, 64, False)])
def test_prompt_chunks_of_few_tokens_take_their_block_lists_token_by_token(n, n_heads, n_kv, d, alone):
    ops = DryOps(torch.bfloat16)
    assert ops.sm_count == 148 and ops.listed_token_by_token(n, n_heads, n_kv, d, 500) == alone


@pytest.mark.parametrize("n,n_heads,n_kv,d,tiles,n_splits", [
    (31, 32, 2, 128, False, None), (32, 32, 2, 128, True, 1), (57, 32, 2, 128, True, 1), (74, 32, 2, 128, True, 1), (75, 32, 2, 128, True, 1),
    (57, 8, 2, 128, False, 1), (31, 16, 2, 64, False, None), (148, 16, 2, 64, False, 1), (149, 16, 2, 64, True, 1)])
def test_the_long_context_shapes_prompts_take_their_block_lists_in_tiles(n, n_heads, n_kv, d, tiles, n_splits):
    """However few their tokens: where many keys weigh alike, a token's own walk has the larger error there."""
    ops, lane, asked = DryOps(torch.bfloat16), SimpleNamespace(k=None, v=None, page_table=torch.empty(1, 500, device="meta")), {}
    ops.listed_attention = lambda *a, **kw: asked.update(kw)
    ctx = SimpleNamespace(is_decode=False, positions=None, token_seq=None, slot_dev=None)
    ops.attention(ctx, torch.empty(n, n_heads, d, device="meta"), lane, n_kv, 1.0, block_list=torch.empty(0), block_size=64)
    assert asked == {"tiles": tiles, "n_splits": n_splits}


@pytest.mark.parametrize("which", ["none", "a", "w"])
def test_the_librarys_per_head_product_takes_operands_that_want_a_gradient(which):
    """Into a view whose matrices lie between each other's rows, as torch's product takes them: the results, and the gradient if one is wanted."""
    g = torch.Generator().manual_seed(3)
    a, w, out = torch.randn(5, 2, 12, generator=g), torch.randn(2, 12, 7, generator=g), torch.zeros(5, 2, 7)
    want = torch.einsum("thk,hkn->thn", a, w)
    for name, t in (("a", a), ("w", w)):
        t.requires_grad_(name == which)
    Ops._library_bmm(SimpleNamespace(), a.transpose(0, 1), w, out.transpose(0, 1))
    assert torch.allclose(out, want, atol=1e-5) and out.requires_grad == (which != "none")
    if which != "none":
        out.sum().backward()
        grad = {"a": w.sum(2).expand(5, 2, 12), "w": a.sum(0)[:, :, None].expand(2, 12, 7)}[which]
        assert torch.allclose({"a": a, "w": w}[which].grad, grad, atol=1e-4)


@pytest.mark.parametrize("rows,longest,shares", [(1, 32000, 16), (6, 32000, 16), (7, 32000, 14), (8, 32000, 12), (9, 32000, 10), (10, 32000, 9),
                                                 (12, 32000, 8), (16, 32000, 6), (20, 32000, 5), (24, 32000, 4), (32, 32000, 4), (8, 4096, 8),
                                                 (16, 4096, 6), (37, 4096, 4), (40, 4096, 1), (75, 4096, 1)])
def test_head_size_64_has_as_many_shares_as_clusters_run_at_once(rows, longest, shares):
    ops = DryOps(torch.bfloat16)
    ops.lib = SimpleNamespace(cpm_decode_attention_blocks_per_sm=lambda d: 2)
    assert ops.decode_splits(rows, 16, 2, 64, longest) == shares


@pytest.mark.parametrize("portions,by_tiles", [
    ([2048], True), ([512], True), ([256], True), ([128], False), ([16], False), ([16] * 64, False), ([32] * 64, False),
    ([1] * 63 + [256], False), ([1] * 63 + [1985], False), ([65] * 15 + [1073], True), ([512] * 4, True), ([8] * 63 + [1544], False),
    ([1] * 255 + [45], False), ([1] * 8 + [504], True),
])
def test_recurrence_goes_by_tiles_where_they_are_few_and_full(portions, by_tiles):
    """Few long portions go by tiles; many short ones, each of which would fill a tile of its own, token by token."""
    ops = DryOps(torch.float32)
    ctx = dry_context(portions, max(portions), None, all(n == 1 for n in portions))
    assert ops.recurrence_by_tiles(ctx, 64, 128) == by_tiles


@pytest.mark.parametrize("portions,keys,by_pairs", [
    ([128], 128, True), ([96], 96, False), ([96], 1096, True), ([95], 4000, False), ([1] * 95 + [2], 1000, False), ([1] * 63 + [1985], 1985, True),
    ([8] * 32, 8, False), ([8] * 32, 1008, True), ([3] * 40, 1003, False), ([1] * 128, 4000, False),
])
def test_latent_attention_goes_by_pairs_where_they_share_keys(portions, keys, by_pairs):
    """Prompt tokens in portions long enough for both tokens of a pair, over histories long enough for the pages they share."""
    ops = DryOps(torch.bfloat16)
    ctx = dry_context(portions, keys, None, all(n == 1 for n in portions))
    assert ops.latent_prompt_ok(ctx, sum(portions)) == by_pairs


@pytest.mark.parametrize("pairs,experts,by_pair", [(160, 64, True), (161, 64, False), (160, 14, True), (160, 13, False), (24, 2, True), (25, 2, False), (12, 1, True)])
def test_experts_go_by_pair_for_few_pairs_and_few_an_expert(pairs, experts, by_pair):
    ops = DryOps(torch.bfloat16)
    assert ops.moe_by_pair(pairs, experts, 64, 32) == by_pair
    assert not ops.moe_by_pair(pairs, experts, 64, 20) and not DryOps(torch.float32).moe_by_pair(pairs, experts, 64, 32)
