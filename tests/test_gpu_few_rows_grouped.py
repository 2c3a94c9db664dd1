"""The grouped product of few rows (routed experts of a step of up to 16 tokens) against the grouped tensor-core product and
64-bit sums."""
from __future__ import annotations

import pytest
import torch

from gpu_util import DEV, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,experts,top", [(1, 16, 2), (3, 5, 1), (8, 16, 2), (8, 4, 4), (9, 7, 3), (16, 1, 1), (16, 64, 6)])
@pytest.mark.parametrize("N,K", [(16, 8), (48, 72), (320, 512), (3072, 2048), (2048, 1536)])
@pytest.mark.parametrize("epilogue,activation", [("plain", None), ("swiglu", None), ("swiglu", ("swish_clamp", 7.0, 0.0))])
def test_few_rows_grouped(n, experts, top, N, K, epilogue, activation):
    """Experts without rows, with one, with all of the step's; sizes around a block's 16 features and a warp's 32 columns.
    32-bit sums of bfloat16 products: 2e-5 of the largest for 32-bit results, a bfloat16 rounding more (2^-8) for gated ones."""
    from nncpu_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(n * experts + K)
    ids = torch.stack([torch.randperm(experts, generator=g, device=DEV)[:top] for _ in range(n)]).to(torch.int32)
    S = n * top
    rows, slots = (torch.empty(S, dtype=torch.int32, device=DEV) for _ in range(2))
    plan = torch.empty(1 + 3 * ops.moe_plan_tiles(S, experts), dtype=torch.int32, device=DEV)
    ops.moe_plan(ids, experts, rows, slots, plan)
    xs = torch.randn(S, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(experts, N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    gated = epilogue == "swiglu"
    dtype = torch.bfloat16 if gated else torch.float32
    out, ref = (torch.full((S, N // 2 if gated else N), 9.0, dtype=dtype, device=DEV) for _ in range(2))
    ops.linear_skinny_grouped(xs, w, out, plan, experts, n, epilogue, activation)
    ops.linear_tc_grouped(xs, w, ref, plan, experts, ops.GemmWorkspace(DEV), epilogue, activation)
    check(out, ref, 2.0 ** -7 if gated else 2e-5, "the tensor-core product")
    if not gated:
        expert = ids.flatten()[slots.long()].long()
        want = torch.einsum("sk,snk->sn", xs.double(), w[expert].double())
        check(out, want.float(), 2e-5, "64-bit sums")


@pytest.mark.parametrize("n,bad,top", [(4, 1, 4), (8, 4, 6), (9, 3, 2), (16, 10, 4)])
def test_tokens_that_are_not_numbers_keep_to_themselves(n, bad, top):
    """A token whose router logits are not numbers chooses expert 0 over and over, so that expert has more rows than the step has
    tokens.  Every row is computed all the same: the other tokens, which choose it too, get the bits they get beside
    healthy tokens, out of memory that held NaN before."""
    from types import SimpleNamespace
    from nncpu_b200.config.specs import RoutedExpertsSpec
    from nncpu_b200.parts import Runtime, base
    from nncpu_b200.parts.runtime import Arena
    width, ff, E = 128, 64, 7
    spec = RoutedExpertsSpec(kind="routed_experts", name="m", hidden_size=width, intermediate_size=ff, n_experts=E, top=top,
                             activation="silu", limit=0.0, router_bias=True)
    part, rt = base.build("feed_forward", spec), Runtime(DEV, torch.bfloat16)
    g = torch.Generator(device=DEV).manual_seed(n)
    tensors = {p.name: (torch.randn(p.shape, generator=g, device=DEV) * 0.1).bfloat16() for p in part.params()}
    tensors["m.router.b"][0] = 50.0                  # everybody's first choice
    part.bind(tensors, rt)
    x = torch.randn(n, width, generator=g, device=DEV).bfloat16()
    outs = []
    for spoilt in (False, True):
        arena = Arena(rt.device)
        arena.reserve(1 << 20)
        arena.buf.fill_(255)
        arena.begin()
        rows = x.clone()
        if spoilt:
            rows[:bad] = float("nan")
        out = torch.zeros(n, width, device=DEV)
        with rt.using(arena):
            part.forward(SimpleNamespace(n_tokens=n), rows, out)
        outs.append(out)
    assert torch.isfinite(outs[0]).all() and not torch.isfinite(outs[1][:bad]).any()
    assert torch.equal(outs[0][bad:], outs[1][bad:])
