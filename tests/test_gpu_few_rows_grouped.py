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
