"""Products of 17 to 256 tokens that run in stripes of the weights: every split of the tokens over blocks and of the weight rows over
SMs, against 64-bit sums."""
import numpy as np
import pytest
import torch

import plain_qwen3 as P

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from nncpu_b200.kernels import ops
    return ops


def near(got, want, rel):
    """rel bounds the largest difference over the result's root mean square; bfloat16 results are off by half a unit in the last
    place (2^-9 of a value; values reach some five times the root mean square)."""
    assert (got.double() - want).abs().max().item() <= rel * want.pow(2).mean().sqrt().item()


def f32(k, factor=1.0):
    """Of float32 results: the tensor core cuts its running sum, not rounds it, once for 16 columns, by up to 2^-23 of what it
    holds: half of the result on the way to it, and the largest results are some five times the root mean square."""
    return factor * (2e-6 + k / 16 * 2.0 ** -23 * 2.5)


# tokens: both ends of the three layouts, odd counts, rows that fill a block or leave one to the second block of a pair
@pytest.mark.parametrize("m", [17, 24, 63, 64, 65, 71, 128, 129, 200, 255, 256])
# features: fewer than a stripe each, ragged, one instruction and two, one round over the SMs and more; columns: one chunk, fewer than a
# stage holds, no multiple of a stage; rows so long that two blocks share them up to 64 tokens, in parts that are not equal
@pytest.mark.parametrize("n,k", [(2050, 64), (2368, 192), (4097, 1088), (9480, 2048), (25008, 320), (76000, 128),
                                 (2050, 5184), (1210, 6208), (80, 5248)])
def test_stripes(ops, m, n, k):
    g = torch.Generator().manual_seed(m * 7 + n + k)
    x = torch.randn(m, k, generator=g).bfloat16().to(DEV)
    w = (torch.randn(n, k, generator=g) * 0.1).bfloat16().to(DEV)
    b = torch.randn(n, generator=g).to(DEV)
    ws = ops.GemmWorkspace(DEV)
    want = x.double() @ w.double().T
    out = torch.full((m, n), 9.0, device=DEV)
    ops.linear_tc(x, w, b, out, ws)
    near(out, want + b.double(), f32(k))
    again = torch.full((m, n), 9.0, device=DEV)
    ops.linear_tc(x, w, b, again, ws)
    assert torch.equal(out, again)
    for dt, rel in ((torch.float32, f32(k)), (torch.bfloat16, 0.02)):
        acc = torch.full((m, n), 0.5, dtype=dt, device=DEV)
        ops.linear_tc(x, w, None, acc, ws, accumulate=True)
        near(acc, want + 0.5, rel)
    act = torch.full((m, n), 9.0, device=DEV)
    ops.linear_tc(x, w, b, act, ws, activation=("relu2", 0.5, 0.0))
    near(act, (want + b.double()).clamp(min=0).pow(2) * 0.5, f32(k, 10))       # a square: twice the relative error, of values up to five times the rms
    if n % 16 == 0:
        gated = torch.full((m, n // 2), 9.0, device=DEV)
        ops.linear_tc(x, w, None, gated, ws, epilogue="swiglu")
        y = want.view(m, n // 16, 2, 8)
        near(gated, (torch.nn.functional.silu(y[:, :, 0]) * y[:, :, 1]).reshape(m, -1), f32(k, 10))
    assert int(ws.status.item()) == 0


@pytest.mark.parametrize("m", [17, 64, 65, 128, 129, 250, 256])
@pytest.mark.parametrize("hidden,inter", [(2048, 2432), (4160, 1088), (1024, 5184)])
def test_stripes_carry_the_norm_between_two_products(ops, m, hidden, inter):
    """The product that adds into the residual stream leaves residual * gamma and the exact sums of squares of its rows; the next one
    applies the rows' scales; the accumulators of the norm before are cleared.  Rows of C need not be 16-byte aligned."""
    g = torch.Generator().manual_seed(m + hidden)
    act = torch.randn(m, inter, generator=g).bfloat16().to(DEV)
    w_down = (torch.randn(hidden, inter, generator=g) * 0.1).bfloat16().to(DEV)
    residual0 = torch.randn(m, hidden, generator=g).to(DEV)
    gamma = (1 + 0.1 * torch.randn(hidden, generator=g)).bfloat16().to(DEV)
    eps, ws = 1e-5, ops.GemmWorkspace(DEV)
    assert ops.linear_tc_norm_roles(m, hidden, inter) == 3
    residual = residual0.clone()
    xg = torch.full((m, hidden), 9.0, dtype=torch.bfloat16, device=DEV)
    bins = torch.zeros(m, ops.NORM_ROW_WORDS, dtype=torch.int64, device=DEV)
    stale = torch.full((m, ops.NORM_ROW_WORDS), 77, dtype=torch.int64, device=DEV)
    ops.linear_tc(act, w_down, None, residual, ws, accumulate=True, norm_out=(xg, gamma, bins, stale))
    plain = residual0.clone()
    ops.linear_tc(act, w_down, None, plain, ws, accumulate=True)
    assert torch.equal(residual, plain) and int(stale.abs().max()) == 0
    assert torch.equal(xg, (residual * gamma.float()).bfloat16())
    words = bins.cpu().numpy().astype(object)
    total = np.array([float(sum(int(words[t][b]) * 2.0 ** (32 * b - 150) for b in range(8))) for t in range(m)])
    want_ss = (residual.double() ** 2).sum(-1).cpu().numpy()
    assert np.abs(total - want_ss).max() <= 1e-6 * want_ss.max() and int(bins[:, 8].sum()) == 0
    normed = torch.from_numpy(P.rmsnorm(residual.cpu().numpy(), gamma.float().cpu().numpy(), eps)).double().to(DEV)
    wide = max(2 * hidden, 4224)                   # with 2^22 weights a product of 65 tokens and more carries the norm before it
    w_next = (torch.randn(wide, hidden, generator=g) * 0.1).bfloat16().to(DEV)
    want = normed @ w_next.double().T
    out = torch.full((m, wide), 9.0, device=DEV)
    ops.linear_tc(xg, w_next, None, out, ws, norm_in=(bins, eps))
    near(out, want, 0.02)                          # x * gamma is rounded to bfloat16 before the product
    gated = torch.full((m, wide // 2), 9.0, device=DEV)
    ops.linear_tc(xg, w_next, None, gated, ws, epilogue="swiglu", norm_in=(bins, eps))
    y = want.view(m, wide // 16, 2, 8)
    near(gated, (torch.nn.functional.silu(y[:, :, 0]) * y[:, :, 1]).reshape(m, -1), 0.1)   # a product of two such numbers, values up to 25 times the rms
    odd = torch.empty(m * hidden + 1, device=DEV)[1:].view(m, hidden)
    odd.copy_(residual0)
    odd_xg, odd_bins = torch.full_like(xg, 9.0), torch.zeros_like(bins)
    ops.linear_tc(act, w_down, None, odd, ws, accumulate=True, norm_out=(odd_xg, gamma, odd_bins, None))
    assert torch.equal(odd, residual) and torch.equal(odd_xg, xg) and torch.equal(odd_bins, bins)
    assert int(ws.status.item()) == 0


@pytest.mark.parametrize("m,n,k", [(64, 2048, 2048), (64, 2048, 6336), (128, 6144, 1344), (256, 6144, 2112)])
def test_a_token_has_the_same_bits_beside_any_others(ops, m, n, k):
    """A stage holds one, two or four chunks of K by the number of tokens; halves of K and its parts that are summed by themselves do
    not depend on that (within 17 to 64, 65 to 128 and 129 to 256 tokens)."""
    g = torch.Generator().manual_seed(n)
    x = torch.randn(m, k, generator=g).bfloat16().to(DEV)
    w = (torch.randn(n, k, generator=g) * 0.1).bfloat16().to(DEV)
    ws = ops.GemmWorkspace(DEV)
    want = torch.empty(m, n, device=DEV)
    ops.linear_tc(x, w, None, want, ws)
    for rows in ((17, 31, 40, 57) if m == 64 else (m // 2 + 1, m // 2 + 20, m - 9)):
        out = torch.empty(rows, n, device=DEV)
        ops.linear_tc(x[:rows].contiguous(), w, None, out, ws)
        assert torch.equal(out, want[:rows]), rows
    assert int(ws.status.item()) == 0


# the first numbers of a size: 2-norm of the error against 64 bits, of the result's, as measured; one accumulator over all of K
# is at 4.4e-6 (K 4096) to 1.4e-5 (K 12288), of gated products, which multiply two such sums, at twice as much
@pytest.mark.parametrize("m,n,k,epilogue,measured", [
    (24, 4096, 4096, "plain", 4.8e-7), (24, 4096, 12288, "plain", 7.4e-7), (64, 4096, 4096, "plain", 4.8e-7),
    (64, 4096, 12288, "plain", 7.4e-7), (64, 4096, 2560, "plain", 2.4e-7), (64, 24576, 4096, "swiglu", 4.3e-6),
    (100, 4096, 4096, "plain", 4.8e-7), (100, 2048, 4096, "plain", 2.5e-7), (100, 4096, 12288, "plain", 1.6e-6),
    (100, 65536, 4096, "plain", 2.2e-6), (200, 4096, 4096, "plain", 4.8e-7), (200, 4096, 12288, "plain", 1.6e-6),
    (200, 24576, 4096, "swiglu", 4.3e-6), (200, 65536, 2048, "plain", 1.0e-6), (200, 1024, 5184, "plain", 2.5e-7)])
def test_sums_are_as_near_to_64_bits_as_without_stripes(ops, m, n, k, epilogue, measured):
    g = torch.Generator(device=DEV).manual_seed(n + k)
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(n, k, generator=g, device=DEV) * 0.02).bfloat16()
    want = x.double() @ w.double().T
    if epilogue == "swiglu":
        y = want.view(m, n // 16, 2, 8)
        want = (torch.nn.functional.silu(y[:, :, 0]) * y[:, :, 1]).reshape(m, -1)
    ws = ops.GemmWorkspace(DEV)
    off = {}
    for plan in ("auto", "no_stripes"):
        out = torch.empty_like(want, dtype=torch.float32)
        ops.linear_tc(x, w, None, out, ws, epilogue=epilogue, plan=plan)
        off[plan] = ((out.double() - want).norm() / want.norm()).item()
    assert ops.linear_tc_stripes(m, n, k, epilogue) is not None
    assert off["auto"] <= 1.25 * measured and off["auto"] <= max(1.03 * off["no_stripes"], 2.6e-7), off
    assert int(ws.status.item()) == 0
