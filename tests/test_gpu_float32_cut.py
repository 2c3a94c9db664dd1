"""Float32 products whose tokens are cut into their parts beforehand: the same bits as cut where they arrive."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("m", [95, 96, 97, 257])
@pytest.mark.parametrize("k", [36, 100, 1092])
def test_tokens_cut_beforehand(m, k):
    """Around the number of tokens from which they are, one beyond a tile of 256, and widths that end inside a block of 32 columns
    and inside eight numbers; numbers of very different sizes, an infinity among them.  Enough features that K stays in one
    slice, so that the product also runs without scratch memory, which cuts on arrival.  64-bit sums: the tensor core sums 64
    columns by itself, 32 below K 512 (3.4e-7 of the 2-norm at most, a quarter more allowed)."""
    from nncpu_b200.kernels import ops
    g = torch.Generator().manual_seed(m + k)
    n = 128 * 148 - 7
    x = (torch.randn(m, k, generator=g) * torch.exp2(torch.randint(-20, 20, (m, 1), generator=g).float())).to(DEV)
    w = (torch.randn(n, k, generator=g) * 0.02).to(DEV)
    bias = torch.randn(n, generator=g).to(DEV)
    work = ops.GemmWorkspace(DEV)
    floats = ops.linear_f32_many_scratch_floats(m, n, k)
    assert floats == (0 if m < 96 else m * ((k + 31) // 32) * 48)
    scratch = torch.full((floats,), float("nan"), device=DEV) if floats else None
    out, other = torch.full((m, n), 9.0, device=DEV), torch.full((m, n), 9.0, device=DEV)
    ops.linear_f32_many(x, w, None, out, scratch, work)
    ops.linear_f32_many(x, w, None, other, None, work)
    assert torch.equal(out, other)
    want = x.double() @ w.double().T
    assert ((out.double() - want).norm(dim=1) / want.norm(dim=1)).max().item() < 4.3e-7
    x[m // 2, k - 1] = float("inf")
    ops.linear_f32_many(x, w, bias, out, scratch, work, accumulate=True)
    ops.linear_f32_many(x, w, bias, other, None, work, accumulate=True)
    assert torch.equal(out, other) and bool(torch.isinf(out[m // 2]).all())
    assert int(work.status.item()) == 0


def test_many_tokens_go_in_bands():
    """The tokens' parts take 256 MB at most; a band has the bits of a product of its own."""
    from nncpu_b200.kernels import ops
    m, n, k, band = 7300, 264, 6144, 3840
    floats = ops.linear_f32_many_scratch_floats(m, n, k)
    assert floats == max(ops.linear_f32_many_scratch_floats(rows, n, k) for rows in (band, m - band)) < m * k * 3 // 2
    g = torch.Generator(device=DEV).manual_seed(5)
    x, w = torch.randn(m, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV) * 0.02
    bias, work = torch.randn(n, generator=g, device=DEV), ops.GemmWorkspace(DEV)
    scratch = torch.full((floats + 1,), 7.0, device=DEV)
    for dtype in (torch.float32, torch.bfloat16):
        out, parts = [torch.full((m, n), 9.0, dtype=dtype, device=DEV) for _ in range(2)]
        ops.linear_f32_many(x, w, bias, out, scratch[:floats], work)
        for rows in (slice(0, band), slice(band, m)):
            ops.linear_f32_many(x[rows], w, bias, parts[rows], scratch[:floats], work)
        assert torch.equal(out, parts) and float(scratch[-1]) == 7.0
        want = x.double() @ w.double().T + bias.double()
        assert ((out.double() - want).norm() / want.norm()).item() < (4.3e-7 if dtype == torch.float32 else 2.0 ** -8)
    assert int(work.status.item()) == 0
