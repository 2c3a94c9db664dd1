"""Decode attention of more blocks than run at once: they may start in the order of their sequences' lengths, and every sequence
has the bits that it has alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from nncpu_b200.kernels import ops
    return ops


@pytest.mark.parametrize("n,nkv", [(1, 8), (37, 8), (38, 8), (75, 4), (127, 4), (128, 8), (129, 4)])
def test_every_sequence_has_the_bits_that_it_has_alone(ops, n, nkv):
    """In the tokens' order and by length; ties, sequences of one key, and padding between them."""
    g = torch.Generator().manual_seed(n)
    heads, hd = 2 * nkv, 64
    pos = torch.randint(0, 300, (n,), generator=g, dtype=torch.int32)
    pos[::5] = 200                                  # ties
    pos[1::7] = 0
    pages = [int(p) // 64 + 1 for p in pos]
    table, at = torch.zeros(n, max(pages), dtype=torch.int32), 0
    for i, k in enumerate(pages):
        table[i, :k] = torch.arange(at, at + k, dtype=torch.int32)
        at += k
    seq = torch.arange(n, dtype=torch.int32)
    seq[3::11] = -1                                 # padding
    k_pages = torch.randn(at, nkv, 64, hd, generator=g).bfloat16().to(DEV)
    v_pages = torch.randn(at, nkv, 64, hd, generator=g).bfloat16().to(DEV)
    q = torch.randn(n, heads * hd, generator=g).bfloat16().to(DEV)
    table, seq, pos = table.to(DEV), seq.to(DEV), pos.to(DEV)
    out = torch.full((n, heads * hd), 9.0, dtype=torch.bfloat16, device=DEV)
    ops.attention_decode_mma(q, k_pages, v_pages, table, seq, pos, out, None, heads, nkv, hd, hd ** -0.5, 0, 1)
    order, by_length = torch.full((n, 4), 9, dtype=torch.int32, device=DEV), torch.full_like(out, 7.0)
    ops.attention_decode_order(seq, pos, order)
    keys = torch.where(seq < 0, -1, pos).cpu()
    want = sorted(range(n), key=lambda i: -int(keys[i]))           # (stable: ties in their order)
    assert order.tolist() == [[i, int(seq[i]), int(keys[i]), 0] for i in want]
    ops.attention_decode_mma(q, k_pages, v_pages, table, seq, pos, by_length, None, heads, nkv, hd, hd ** -0.5, 0, 1, order=order)
    assert torch.equal(out, by_length)
    for t in range(n):
        one = torch.full((1, heads * hd), 5.0, dtype=torch.bfloat16, device=DEV)
        ops.attention_decode_mma(q[t:t + 1].contiguous(), k_pages, v_pages, table, seq[t:t + 1].contiguous(), pos[t:t + 1].contiguous(),
                                 one, None, heads, nkv, hd, hd ** -0.5, 0, 1)
        assert torch.equal(out[t], one[0]), t


@pytest.mark.parametrize("n", [1, 255, 257, 1000, 1024])
def test_order_of_many_tokens(ops, n):
    g = torch.Generator().manual_seed(n)
    pos = torch.randint(0, n // 2 + 1, (n,), generator=g, dtype=torch.int32)
    seq = torch.where(torch.rand(n, generator=g) < 0.1, -1, torch.arange(n)).int()
    order = torch.empty(n, 4, dtype=torch.int32, device=DEV)
    ops.attention_decode_order(seq.to(DEV), pos.to(DEV), order)
    keys = torch.where(seq < 0, -1, pos)
    assert order[:, 0].tolist() == sorted(range(n), key=lambda i: -int(keys[i]))
