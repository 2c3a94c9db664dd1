"""Products on pairs of SMs whose tiles are walked through in bands of rows: the order of the tiles is no part of a result, so a
product of many rows has the bits of the products of its pieces, each of which is one band."""
from __future__ import annotations

import pytest
import torch

from gpu_util import DEV, check

pytestmark = pytest.mark.gpu

# rows: one band less a row, 9 tile rows (bands of 5 and 4), 11 (6 and 5), 16 (8 and 8), 17 (6, 6 and 5), 20 (7, 7 and 6)
ROWS = [2047, 2304, 2561, 4096, 4352, 4866]


@pytest.fixture(scope="module")
def ops():
    from nncpu_b200.kernels import ops
    return ops


def pieces(m):
    """Row ranges of 512 to 2 048 rows (eight tile rows at most, and enough for this kernel)."""
    cuts = list(range(0, m - 511, 1024)) + [m]
    return [slice(a, b) for a, b in zip(cuts, cuts[1:])]


@pytest.mark.parametrize("m", ROWS)
@pytest.mark.parametrize("n,k", [(512, 64), (777, 264), (2560, 128)])
def test_plain_and_gated(ops, m, n, k):
    """One column of tiles and several, a ragged last one, against the pieces and against 64-bit sums (32-bit sums of bfloat16
    products: 1e-5 of the largest)."""
    g = torch.Generator(device=DEV).manual_seed(m + n)
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(n, k, generator=g, device=DEV) * 0.1).bfloat16()
    b = torch.randn(n, generator=g, device=DEV)
    ws = ops.GemmWorkspace(DEV)
    out, part = (torch.full((m, n), 9.0, device=DEV) for _ in range(2))
    ops.linear_tc(x, w, b, out, ws)
    for r in pieces(m):
        ops.linear_tc(x[r], w, b, part[r], ws)
    assert torch.equal(out, part)
    check(out, (x.double() @ w.double().T + b).float(), 1e-5, "against 64-bit sums")
    if n % 16 == 0:
        out, part = (torch.full((m, n // 2), 9.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        ops.linear_tc(x, w, None, out, ws, epilogue="swiglu")
        for r in pieces(m):
            ops.linear_tc(x[r], w, None, part[r], ws, epilogue="swiglu")
        assert torch.equal(out, part)
    assert int(ws.status.item()) == 0


@pytest.mark.parametrize("m", ROWS)
def test_norms_that_ride_on_them(ops, m):
    """The producer's rows times gamma, its exact accumulators and those it clears, and the consumer's scaled results."""
    g = torch.Generator(device=DEV).manual_seed(m)
    hidden, inter = 1024, 768
    act = torch.randn(m, inter, generator=g, device=DEV).bfloat16()
    w_down = (torch.randn(hidden, inter, generator=g, device=DEV) * 0.1).bfloat16()
    w_next = (torch.randn(inter, hidden, generator=g, device=DEV) * 0.1).bfloat16()
    gamma = (1 + 0.1 * torch.randn(hidden, generator=g, device=DEV)).bfloat16()
    residual = torch.randn(m, hidden, generator=g, device=DEV)
    ws = ops.GemmWorkspace(DEV)
    assert ops.linear_tc_norm_roles(m, hidden, inter) == 3 and ops.linear_tc_norm_roles(m, inter, hidden) == 3

    def run(rows):
        out = torch.empty_like(residual)
        xg = torch.full((m, hidden), 9.0, dtype=torch.bfloat16, device=DEV)
        bins = torch.zeros(m, ops.NORM_ROW_WORDS, dtype=torch.int64, device=DEV)
        stale = torch.full_like(bins, 77)
        nxt = torch.full((m, inter), 9.0, device=DEV)
        for r in rows:
            out[r] = residual[r]
            ops.linear_tc(act[r], w_down, None, out[r], ws, accumulate=True, norm_out=(xg[r], gamma, bins[r], stale[r]))
            ops.linear_tc(xg[r], w_next, None, nxt[r], ws, norm_in=(bins[r], 1e-5))
        return out, xg, bins, stale, nxt

    whole, parts = run([slice(0, m)]), run(pieces(m))
    assert all(torch.equal(a, b) for a, b in zip(whole, parts))
    out, xg, bins, stale, nxt = whole
    assert int(stale.abs().max()) == 0 and int(ws.status.item()) == 0
    normed = out.double() / ((out.double() ** 2).mean(-1, keepdim=True) + 1e-5).sqrt() * gamma.double()
    check(nxt, normed @ w_next.double().T, 8e-3, "consumer")


@pytest.mark.parametrize("m", ROWS)
def test_the_projection_with_its_epilogue(ops, m):
    """q, and the keys and values in their pages."""
    g = torch.Generator(device=DEV).manual_seed(m)
    nh, nkv, hd, k = 6, 2, 128, 128
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn((nh + 2 * nkv) * hd, k, generator=g, device=DEV) * 0.1).bfloat16()
    qg, kg = ((1 + 0.1 * torch.randn(hd, generator=g, device=DEV)).bfloat16() for _ in range(2))
    angle = torch.rand(hd // 2, m, generator=g, device=DEV) * 6
    cs = torch.stack([angle.cos(), angle.sin()], dim=-1).contiguous()
    ws = ops.GemmWorkspace(DEV)
    assert ops.linear_tc_qkv_supported(x, nh, nkv, hd)
    n_pages = (m + 63) // 64
    table = torch.randperm(n_pages, generator=g, device=DEV).to(torch.int32).view(1, -1)
    seq, pos = torch.zeros(m, dtype=torch.int32, device=DEV), torch.arange(m, dtype=torch.int32, device=DEV)

    def run(rows):
        kp, vp = (torch.zeros(n_pages, nkv, 64, hd, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        q = torch.full((m, nh * hd), 9.0, dtype=torch.bfloat16, device=DEV)
        for r in rows:
            ops.linear_tc_qkv(x[r], w, qg, kg, 1e-6, cs[:, r].contiguous(), seq[r], pos[r], table, kp, vp, q[r], ws, nh, nkv, hd)
        return q, kp, vp

    whole, parts = run([slice(0, m)]), run(pieces(m))
    assert all(torch.equal(a, b) for a, b in zip(whole, parts)) and int(ws.status.item()) == 0
    v = (x.double() @ w[(nh + nkv) * hd:].double().T).view(m, nkv, hd)
    got = whole[2][table[0].long()].transpose(1, 2).reshape(-1, nkv, hd)[:m]
    check(got, v, 8e-3, "values")
