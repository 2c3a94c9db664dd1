"""Norms of few and of many rows: weights that are not 16-byte aligned, every width's kernel, and 64-bit values."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from nncpu_b200.kernels import ops
    return ops


def norm(x, gamma, eps=1e-6):
    x = x.double()
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * gamma.double()


# rows: one, and around two and four an SM; lanes: the ends of each kernel's widths
@pytest.mark.parametrize("rows", [1, 296, 297, 592, 593])
@pytest.mark.parametrize("dim", [1024, 1028, 2048, 2052, 4096, 4100, 8192])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norms_whatever_the_alignment_of_the_weights(ops, rows, dim, dtype):
    """The same bits with weights that a thread reads four at a time and one by one; sums of at most 32 numbers a thread and of 256
    threads in float32, three factors: 1e-6 of a value, of whose rounding to bfloat16 there is nothing here."""
    g = torch.Generator(device=DEV).manual_seed(rows + dim)
    x, r = torch.randn(rows, dim, generator=g, device=DEV), torch.randn(rows, dim, generator=g, device=DEV)
    weights = (1 + 0.1 * torch.randn(2, dim, generator=g, device=DEV)).to(dtype)
    results = []
    for off in (0, 1):
        g1, g2 = (torch.empty(dim + 8, dtype=dtype, device=DEV)[off:off + dim].copy_(w) for w in weights)
        assert (g1.data_ptr() % 16 == 0) == (off == 0)
        one, two, y1, y2 = (torch.empty(rows, dim, device=DEV) for _ in range(4))
        added, stream = r.clone(), r.clone()
        ops.rmsnorm(x, g1, 1e-6, one)
        ops.rmsnorm(x, g1, 1e-6, added, accumulate=True)
        ops.rmsnorm_pair(x, stream, g1, 0.0, 1e-6, g2, 0.0, 1e-6, two)
        ops.rmsnorm_dual(x, g1, 1e-6, g2, 1e-6, y1, y2)
        results.append((one, added, stream, two, y1, y2))
    assert all(torch.equal(a, b) for a, b in zip(*results))
    first, second = norm(x, weights[0]), norm(x, weights[1])
    sums = r.double() + first
    for got, want in zip(results[0], (first, sums, sums, norm(sums, weights[1]), first, second)):
        assert ((got.double() - want).abs() <= 1e-6 * (want.abs() + 1)).all()
