"""Rules that choose a kernel by sizes alone, without a GPU."""
from __future__ import annotations

from types import SimpleNamespace

import pytest

from nncpu_b200.kernels import ops
from nncpu_b200.parts.attention import Attention


@pytest.mark.parametrize("n_seqs,tokens,n_kv,window,longest,few", [
    (1, 24, 4, 0, 724, True), (1, 24, 4, 0, 4096, False),      # by the keys there may be
    (1, 16, 8, 0, 4096, True), (1, 16, 8, 0, 4700, False), (1, 17, 8, 0, 4096, False),
    (1, 64, 4, 0, 300, True), (1, 64, 8, 0, 65, False),        # by the blocks
    (1, 32, 8, 0, 100, True), (1, 33, 8, 0, 100, False),
    (1, 24, 4, 512, 40960, True),                              # a window bounds the keys
    (2, 24, 4, 0, 100, False), (1, 65, 1, 0, 100, False)])
def test_short_portions_token_by_token(n_seqs, tokens, n_kv, window, longest, few):
    part = Attention.__new__(Attention)
    part.spec = SimpleNamespace(n_kv_heads=n_kv, window=window, keep_first=0, chunk=0)
    assert part._few_over_short(SimpleNamespace(n_seqs=n_seqs, n_tokens=tokens, max_kv_len=longest)) is few


@pytest.mark.parametrize("tokens,decode,n_seqs,by_token", [
    (1, True, 1, True), (500, True, 500, True), (2, False, 1, True), (64, False, 1, True), (65, False, 1, False),
    (83, False, 64, True),                  # decode rows beside a portion
    (192, False, 64, True), (256, False, 64, True), (257, False, 64, False), (331, False, 32, False)])
def test_float32_attention_token_by_token(tokens, decode, n_seqs, by_token):
    chunk, stretches = ops.attention_f32_plan(tokens, decode, 700, n_seqs)
    assert (chunk > 0) is by_token and (stretches * chunk >= 700 or tokens > 64 or not by_token)


@pytest.mark.parametrize("m,n,k,pays", [
    (1, 1024, 1024, True), (1, 1023, 1024, False), (300, 1023, 1024, False), (300, 1024, 1024, True),
    (1, 4096, 256, True), (4, 150000, 252, False), (5, 150000, 512, False), (16, 150000, 640, True),
    (17, 65536, 32, False), (17, 21856, 48, True), (1, 65536, 16, False)])
def test_float32_products(m, n, k, pays):
    assert ops.linear_f32_pays(m, n, k) is pays


@pytest.mark.parametrize("tokens,top,pays", [(8, 2, True), (16, 4, True), (8, 8, True), (16, 5, False), (9, 8, False), (17, 1, False)])
def test_routed_experts_by_the_few_row_product(tokens, top, pays):
    assert ops.skinny_grouped_pays(tokens, tokens * top) is pays


@pytest.mark.parametrize("m", [95, 96, 3000, 7281, 7282, 8192, 20000, 100000])
@pytest.mark.parametrize("n,k", [(2048, 6144), (12288, 2048), (256, 17408), (128, 100000)])
def test_float32_parts_are_bounded(m, n, k):
    """The scratch of float32 products of many tokens: the tokens' parts, in bands of 2^26 floats (and less than 256 tokens more), and
    the sums of K's slices where there are few tiles."""
    blocks = (k + 31) // 32 * 48
    most = min(m, (1 << 26) // blocks + 256)
    assert ops.linear_f32_many_scratch_floats(m, n, k) <= (most * blocks if m >= 96 else 0) + 8 * most * n


@pytest.mark.parametrize("n,heads,n_kv,k_row,v_row,splits,pays", [
    (37, 32, 8, 128, 128, 1, False), (38, 32, 8, 128, 128, 1, True), (19, 32, 8, 128, 128, 2, True),        # two blocks an SM
    (55, 16, 8, 128, 64, 1, False), (56, 16, 8, 128, 64, 1, True), (74, 16, 8, 64, 64, 1, False), (75, 16, 8, 64, 64, 1, True),
    (74, 64, 1, 128, 128, 1, False), (75, 64, 1, 128, 128, 1, True),                                        # four blocks share a key/value head
    (1024, 32, 8, 128, 128, 1, True), (1025, 32, 8, 128, 128, 1, False)])
def test_decode_blocks_start_by_length(n, heads, n_kv, k_row, v_row, splits, pays):
    assert ops.attention_decode_order_pays(n, heads, n_kv, k_row, v_row, splits, 148) is pays
