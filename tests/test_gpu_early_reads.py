"""Kernels that start under the end of the kernel before them may ask early only for what that one cannot be writing: here the kernel
before writes the weights (it starts its successor at once and then streams some hundred megabytes)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
LONG = 262144
WIDTH = 1024         # results a row of the slow product: 64 blocks, beside which the next kernel finds free SMs


@pytest.fixture(scope="module")
def ops():
    from nncpu_b200.kernels import ops
    return ops


@pytest.fixture(scope="module")
def slow():
    """Operands of a few-token product that takes long for few results."""
    g = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(16, LONG, generator=g, device=DEV, dtype=torch.bfloat16)
    w = (torch.randn(4096, LONG, generator=g, device=DEV, dtype=torch.bfloat16) * 2.0 ** -9)
    return x, w


def both(write, read, target):
    """read() right behind write() into a target that holds something else, and after everything is over."""
    write()
    read()                 # (everything is loaded)
    target.fill_(3.0)
    torch.cuda.synchronize()
    write()
    got = read()
    torch.cuda.synchronize()
    want = read()
    torch.cuda.synchronize()
    return got, want


@pytest.mark.parametrize("m", [65, 100, 128, 129, 200, 256])
def test_stripes_of_weights_just_written(ops, slow, m):
    x, w = slow
    weights = torch.empty(16, WIDTH, dtype=torch.bfloat16, device=DEV)
    act = torch.randn(m, WIDTH, device=DEV).bfloat16()
    ws, outs = ops.GemmWorkspace(DEV), [torch.empty(m, 16, device=DEV) for _ in range(3)]

    def read():
        out = outs.pop()
        ops.linear_tc(act, weights, None, out, ws)
        return out

    got, want = both(lambda: ops.linear_skinny(x, w[:WIDTH], None, weights), read, weights)
    assert ops.linear_tc_stripes(m, 16, WIDTH) is not None and torch.equal(got, want) and int(ws.status.item()) == 0


@pytest.mark.parametrize("m", [96, 300])
def test_float32_product_of_weights_just_written(ops, slow, m):
    x, w = slow
    weights = torch.empty(16, WIDTH, device=DEV)
    act = torch.randn(m, WIDTH, device=DEV)
    floats = ops.linear_f32_many_scratch_floats(m, 16, WIDTH)
    scratch, ws = torch.empty(floats, device=DEV), ops.GemmWorkspace(DEV)
    outs = [torch.empty(m, 16, device=DEV) for _ in range(3)]

    def read():
        out = outs.pop()
        ops.linear_f32_many(act, weights, None, out, scratch, ws)
        return out

    got, want = both(lambda: ops.linear_skinny(x, w[:WIDTH], None, weights), read, weights)
    assert torch.equal(got, want) and int(ws.status.item()) == 0


@pytest.mark.parametrize("dim", [1024, 2048, 4096])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind", ["one", "pair", "dual"])
def test_norm_with_weights_just_written(ops, slow, kind, dtype, dim):
    x, w = slow
    gammas = torch.empty(2, dim, dtype=dtype, device=DEV)
    rows, stream = torch.randn(3, dim, device=DEV), torch.randn(3, dim, device=DEV)
    outs = [[torch.empty(3, dim, device=DEV) for _ in range(2)] for _ in range(3)]
    streams = [stream.clone() for _ in range(3)]

    def read():
        out, r = outs.pop(), streams.pop()
        if kind == "one":
            ops.rmsnorm(rows, gammas[1], 1e-6, out[0])
            out[1].zero_()
        elif kind == "pair":
            ops.rmsnorm_pair(rows, r, gammas[0], 0.0, 1e-6, gammas[1], 0.0, 1e-6, out[0])
            out[1].copy_(r)
        else:
            ops.rmsnorm_dual(rows, gammas[0], 1e-6, gammas[1], 1e-6, out[0], out[1])
        return torch.stack(out)

    got, want = both(lambda: ops.linear_skinny(x[:2], w[:dim], None, gammas), read, gammas)
    assert torch.equal(got, want)
