"""The kernels around latent attention's projections: a few tokens, whose parts and heads several blocks share, give the bits that
the same tokens give in a long prompt, where one block does a token."""
from __future__ import annotations

import pytest
import torch

from gpu_util import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,hd,rank,rot,pairs,q_rank,q_size", [(32, 64, 64, 64, 32, 1536, 0), (5, 24, 40, 16, 6, 72, 0),
                                                                   (16, 128, 128, 0, 0, 0, 2048), (3, 10, 20, 0, 0, 0, 30)])
def test_few_tokens_give_the_bits_of_many(heads, hd, rank, rot, pairs, q_rank, q_size):
    from nncpu_b200.kernels import ops
    n, g = 700, torch.Generator(device=DEV).manual_seed(heads)
    proj = torch.randn(n, q_rank + q_size + rank + rot, generator=g, device=DEV)
    q = torch.randn(n, heads * (hd + rot), generator=g, device=DEV)
    gamma, q_gamma = torch.randn(rank, generator=g, device=DEV), torch.randn(max(q_rank, 1), generator=g, device=DEV)
    cs = torch.randn(n, pairs, 2, generator=g, device=DEV) if pairs else None
    table = torch.arange(11, dtype=torch.int32, device=DEV).view(1, 11)

    def run(lo, hi, pages):
        m = hi - lo
        seq, pos = torch.zeros(m, dtype=torch.int32, device=DEV), torch.arange(lo, hi, dtype=torch.int32, device=DEV)
        c = None if cs is None else cs[lo:hi].contiguous()
        cq = torch.empty(m, q_rank, dtype=torch.bfloat16, device=DEV) if q_rank else None
        qo = torch.empty(m, q_size, dtype=torch.bfloat16, device=DEV) if q_size else None
        ops.latent_append(proj[lo:hi].contiguous(), q_rank + q_size, gamma, 1e-6, seq, pos, table, pages, qo, rot, c,
                          (q_gamma, 0, q_rank, cq) if q_rank else None)
        q_lat = torch.zeros(m, heads * (rank + rot), dtype=torch.bfloat16, device=DEV)
        q16 = torch.empty(m, heads * (hd + rot), dtype=torch.bfloat16, device=DEV)
        ops.latent_query(q[lo:hi].contiguous(), c, q_lat, heads, hd, rot, rank, q16)
        return [t for t in (cq, qo, q_lat, q16) if t is not None]

    pages = [torch.zeros(11, 1, 64, rank + rot, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    whole = run(0, n, pages[0])
    lo = 0
    for m in (1, 2, 16, 64, 98, 99, 420):
        for got, want in zip(run(lo, lo + m, pages[1]), whole):
            assert torch.equal(got, want[lo:lo + m])
        lo += m
    assert lo == n and torch.equal(pages[0], pages[1])
    assert torch.equal(whole[-1], q.bfloat16())
