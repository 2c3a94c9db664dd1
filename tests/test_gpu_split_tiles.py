"""Prompt attention whose tiles of query rows share their keys among the blocks of a cluster, against the same tiles walked by one
block and against the general 32-bit kernel."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from gpu_util import DEV, check, scatter_pages

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from nncpu_b200.kernels import ops
    return ops


@pytest.mark.parametrize("nh,nkv,hd,vd", [(4, 1, 128, 128), (3, 1, 128, 128), (2, 2, 64, 64), (4, 1, 64, 64), (4, 2, 128, 64)])
@pytest.mark.parametrize("how", [dict(), dict(window=100), dict(window=130, keep=9), dict(window=-64), dict(slope_base=8.0),
                                 dict(cap=5.0), dict(sinks=True), dict(head_gate=True), dict(v_lanes=50)], ids=str)
def test_split_tiles(ops, nh, nkv, hd, vd, how):
    """Pasts of many steps, of one, of none (blocks without a step), a span that ends one key into a step, rows that see no key of
    a block's part (windows), a tile and a row: 2, 4 and 8 blocks.  The weights are rounded to bfloat16 against a reference
    that each block keeps for itself: a rounding of 2^-9 of a weight, hence the tolerance of the kernel's other tests."""
    old, new = [700, 0, 127, 1000], [24, 40, 2, 130]
    seqs = [o + n for o, n in zip(old, new)]
    kp, _, table, _, _ = scatter_pages(40, nkv, hd, seqs, torch.bfloat16, seed=nh)
    vp, _, _, _, _ = scatter_pages(40, nkv, vd, seqs, torch.bfloat16, seed=nh)
    n = sum(new)
    tok_seq = [b for b, m in enumerate(new) for _ in range(m)]
    pos = [o + i for o, m in zip(old, new) for i in range(m)]
    g = torch.Generator().manual_seed(5)
    q = torch.randn(n, nh * hd, generator=g).bfloat16()
    how = dict(how)
    window, lanes = how.pop("window", 0), how.get("v_lanes", vd)
    how["v_lanes"] = lanes
    if how.get("sinks"):
        how["sinks"] = torch.randn(nh, generator=g).to(DEV)
    if how.get("head_gate"):
        how["head_gate"] = (torch.randn(n, nh + 3, generator=g).to(DEV), 2)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(new)]).astype(np.int32)).to(DEV)
    tok_pos = torch.tensor(pos, dtype=torch.int32).to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    outs = {}
    for longest in (0, 256, 512, 1130, 40000):
        outs[longest] = torch.full((n, nh * lanes), 9.0, dtype=torch.bfloat16, device=DEV)
        ops.attention_prefill_tc(q.to(DEV), kp, vp, table, cu, tok_pos, outs[longest], status, len(new), nh, nkv, hd,
                                 1 / math.sqrt(hd), window, longest=longest, **how)
    assert int(status.item()) == 0
    for longest, out in outs.items():
        check(out, outs[0], 1.5e-2, f"longest {longest}")
    assert torch.equal(outs[1130], outs[40000])        # both are eight blocks
    want = torch.empty(n, nh * lanes, dtype=torch.bfloat16, device=DEV)
    seq = torch.tensor(tok_seq, dtype=torch.int32).to(DEV)
    ops.attention(q.to(DEV), kp, vp, table, seq, tok_pos, want, nh, nkv, hd, 1 / math.sqrt(hd), window, v_head_dim=vd, **how)
    check(outs[1130], want, 1.5e-2, "the 32-bit kernel")


@pytest.mark.parametrize("nh,nkv,new,longest,splits", [(4, 1, [24], 512, 1), (4, 1, [24], 700, 4), (4, 1, [24], 2000, 8),
                                                       (32, 8, [40, 300], 2000, 2), (32, 8, [128] * 20, 2000, 1)])
def test_how_many_blocks_share_a_tile(ops, nh, nkv, new, longest, splits):
    """As many as have a step of the longest walk each while all clusters run at once; and a tile that has few steps is walked by one
    block, with the bits of a step that shares nothing, whatever the step's longest walk may be."""
    from nncpu_b200.kernels import library
    lib = library.load("attention_tc")
    assert lib.nncpu_attention_prefill_tc_splits(nh, nkv, 128, 128, 0, sum(new), len(new), longest) == splits
    past = [0 if i % 2 else 1800 for i in range(len(new))]         # every other sequence starts: few steps
    seqs = [p + m for p, m in zip(past, new)]
    kp, vp, table, _, _ = scatter_pages(sum((s + 63) // 64 for s in seqs), nkv, 128, seqs, torch.bfloat16, seed=nh)
    n = sum(new)
    q = torch.randn(n, nh * 128, generator=torch.Generator().manual_seed(5)).bfloat16().to(DEV)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(new)]).astype(np.int32)).to(DEV)
    pos = torch.tensor([p + i for p, m in zip(past, new) for i in range(m)], dtype=torch.int32).to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(longest):
        out = torch.full((n, nh * 128), 9.0, dtype=torch.bfloat16, device=DEV)
        ops.attention_prefill_tc(q, kp, vp, table, cu, pos, out, status, len(new), nh, nkv, 128, 128 ** -0.5, 0, longest=longest)
        return out
    alone, shared = run(0), run(longest)
    assert int(status.item()) == 0
    check(shared, alone, 1.5e-2, "shared")
    for i in range(len(new)):
        rows = slice(int(cu[i]), int(cu[i + 1]))
        if i % 2 or splits == 1:
            assert torch.equal(shared[rows], alone[rows])
        else:
            assert not torch.equal(shared[rows], alone[rows])      # several references and orders of sums: other roundings
