"""The kernels of true float32 runs: the products of few and of many tokens, and attention over float32 pages, against 64-bit sums and
against the general kernels."""
from __future__ import annotations

import math

import pytest
import torch

from gpu_util import DEV, check, scatter_pages

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from nncpu_b200.kernels import ops
    return ops


def bound(x, w, extra=4):
    """Largest error that a 32-bit sum of k products in any order may have: (k + extra) roundings of 2^-24 of the sum of the
    products' magnitudes."""
    return (x.shape[1] + extra) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(1, 4), (7, 124), (64, 128), (37, 132), (130, 516), (96, 2048), (33, 6144)])
def test_few_token_product(ops, m, n, k):
    g = torch.Generator(device=DEV).manual_seed(m * n + k)
    x, w, b = (torch.randn(s, generator=g, device=DEV) for s in ((m, k), (n, k), (n,)))
    assert ops.linear_f32_supported(x, w)
    want, tol = x.double() @ w.double().T, bound(x, w) + 1e-6
    out = torch.full((m, n), 7.0, device=DEV)
    ops.linear_f32(x, w, b, out)
    assert ((out - (want + b)).abs() <= tol + b.abs() * 2.0 ** -23).all()
    ops.linear_f32(x, w, None, out, accumulate=True)
    assert ((out - (2 * want + b)).abs() <= 3 * tol + b.abs() * 2.0 ** -22).all()
    half = torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
    ops.linear_f32(x, w, b.bfloat16(), half)
    assert ((half - (want + b.bfloat16())).abs() <= tol + 2.0 ** -8 * (want + b.bfloat16()).abs()).all()
    # a row's result does not depend on the rows beside it
    one = torch.empty(1, n, device=DEV)
    many = torch.empty(16, n, device=DEV)
    ops.linear_f32(x[m - 1:].contiguous(), w, None, one)
    ops.linear_f32(x[m - 1:].expand(16, k).contiguous(), w, None, many)
    assert torch.equal(one.expand(16, n), many)


@pytest.mark.parametrize("m", [1, 17, 32, 33, 64, 90, 128, 160, 190, 224, 256, 257, 300, 520])
@pytest.mark.parametrize("n,k", [(5, 4), (128, 32), (129, 36), (200, 100), (201, 1000), (300, 1000), (1536, 2048), (256, 6144)])
def test_many_token_product(ops, m, n, k):
    """On the tensor cores with numbers cut in three: the bound of a 32-bit sum holds, and over longer sums the error is no
    larger than that of the general kernel, which adds k products one after the other."""
    g = torch.Generator(device=DEV).manual_seed(m * n + k)
    x, w, b = (torch.randn(s, generator=g, device=DEV) for s in ((m, k), (n, k), (n,)))
    want, tol = x.double() @ w.double().T, bound(x, w) + 1e-6
    floats = ops.linear_f32_many_scratch_floats(m, n, k)
    scratch = torch.full((floats,), float("nan"), device=DEV) if floats else None
    work = ops.GemmWorkspace(DEV)
    out = torch.full((m, n), 7.0, device=DEV)
    ops.linear_f32_many(x, w, b, out, scratch, work)
    assert ((out - (want + b)).abs() <= tol + b.abs() * 2.0 ** -23).all()
    ops.linear_f32_many(x, w, None, out, scratch, work, accumulate=True)
    assert ((out - (2 * want + b)).abs() <= 3 * tol + b.abs() * 2.0 ** -22).all()
    ops.linear_f32_many(x, w, None, out, scratch, work)
    again, general = torch.empty_like(out), torch.empty_like(out)
    ops.linear_f32_many(x, w, None, again, scratch, work)
    ops.linear_simt(x, w, None, general)
    assert torch.equal(out, again) and int(work.status.item()) == 0
    if k >= 1000 and m >= 17:
        assert (out - want).norm() <= (general - want).norm()
    half = torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
    ops.linear_f32_many(x, w, b.bfloat16(), half, scratch, work)
    assert ((half - (want + b.bfloat16())).abs() <= tol + 2.0 ** -8 * (want + b.bfloat16()).abs()).all()


def test_many_token_product_of_numbers_at_the_edges(ops):
    """Infinities, numbers next to the largest and NaN give what float arithmetic gives; tiny and huge scales keep their bits."""
    m, n, k = 40, 1100, 1024
    g = torch.Generator(device=DEV).manual_seed(4)
    x, w = torch.randn(m, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV)
    for scale_x, scale_w in ((1e18, 1e18), (1e-12, 1e-12), (1e30, 1e-30)):
        a, b = x * scale_x, w * scale_w
        floats = ops.linear_f32_many_scratch_floats(m, n, k)
        scratch = torch.empty(floats, device=DEV) if floats else None
        out = torch.empty(m, n, device=DEV)
        ops.linear_f32_many(a, b, None, out, scratch, ops.GemmWorkspace(DEV))
        assert ((out - a.double() @ b.double().T).abs() <= bound(a, b)).all()
    x[3, 700], w[5, 9], w[6, 10], x[8, 20], w[11, 20] = math.inf, -math.inf, math.nan, 3.4028234e38, 1.0
    w[:, 700] = w[:, 700].abs()
    got, want = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)
    ops.linear_f32_many(x, w, None, got, scratch, ops.GemmWorkspace(DEV))
    ops.linear_simt(x, w, None, want)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[got.isinf()], want[want.isinf()])
    assert want.isinf().any() and want.isnan().any()


def test_few_token_product_of_other_forms_stays_general(ops):
    x, w = torch.randn(4, 128, device=DEV), torch.randn(8, 128, device=DEV)
    assert not ops.linear_f32_supported(x.bfloat16(), w) and not ops.linear_f32_supported(x, w.bfloat16())
    assert not ops.linear_f32_supported(x[:, :126].contiguous(), w[:, :126].contiguous())
    shifted = torch.randn(8 * 128 + 1, device=DEV)[1:].view(8, 128)
    assert not ops.linear_f32_supported(x, shifted)


def run_attention(ops, q, kp, vp, table, tok_seq, tok_pos, nh, nkv, hd, vd, vo, plan, **how):
    out = torch.full((q.shape[0], nh * vo), 9.0, device=DEV)
    scratch = torch.full((q.shape[0] * nh * plan[1] * (vd + 2),), float("nan"), device=DEV) if plan[1] > 1 else None
    ops.attention_f32(q, kp, vp, table, tok_seq, tok_pos, out, scratch, nh, nkv, hd, 1 / math.sqrt(hd), plan, 148,
                      v_head_dim=vd, v_lanes=vo, **how)
    return out


@pytest.mark.parametrize("nh,nkv,hd,vd,vo", [(4, 4, 128, 128, 128), (2, 1, 64, 64, 64), (6, 2, 16, 36, 20), (4, 1, 128, 64, 64),
                                             (16, 2, 4, 4, 4), (9, 1, 100, 128, 100), (32, 1, 48, 48, 48)])
@pytest.mark.parametrize("how", [dict(), dict(window=50), dict(window=70, keep=5), dict(window=-64), dict(slope_base=8.0),
                                 dict(cap=5.0), dict(sinks=True), dict(head_gate=True)], ids=str)
def test_attention_against_the_general_kernel(ops, nh, nkv, hd, vd, vo, how):
    """Token by token, in every cut of the keys, and in tiles of query rows: lengths at the edges of pages and stretches,
    portions behind a past, a padding row.  Both kernels' softmax weights and sums are 32-bit; 700 keys leave 2e-5 at most."""
    seqs = [700, 1, 64, 65, 128, 129, 300]
    kp, _, table, _, _ = scatter_pages(32, nkv, hd, seqs, torch.float32, seed=hd)
    vp, _, _, _, _ = scatter_pages(32, nkv, vd, seqs, torch.float32, seed=hd)
    g = torch.Generator().manual_seed(nh)
    # the last tokens of every sequence, in order; a padding row between two of them
    tok = [(0, p) for p in range(663, 700)] + [(1, 0)] + [(2, p) for p in range(64)] + [(3, 64), (-1, 3)] + \
        [(4, p) for p in range(120, 128)] + [(5, 127), (5, 128)] + [(6, p) for p in range(300)]
    tok_seq = torch.tensor([t[0] for t in tok], dtype=torch.int32, device=DEV)
    tok_pos = torch.tensor([t[1] for t in tok], dtype=torch.int32, device=DEV)
    q = torch.randn(len(tok), nh * hd, generator=g).to(DEV)
    how = dict(how)
    if how.get("sinks"):
        how["sinks"] = torch.randn(nh, generator=g).to(DEV)
    if how.get("head_gate"):
        how["head_gate"] = (torch.randn(len(tok), nh + 3, generator=g).to(DEV), 2)
    want = torch.empty(len(tok), nh * vo, device=DEV)
    ops.attention(q, kp, vp, table, tok_seq, tok_pos, want, nh, nkv, hd, 1 / math.sqrt(hd), v_head_dim=vd, v_lanes=vo, **how)
    assert ops.attention_f32_supported(q, kp, vp, want, nh, nkv, hd, vd, vo)
    for plan in ((0, 0), (128, 6), (256, 3), (1024, 1)):
        got = run_attention(ops, q, kp, vp, table, tok_seq, tok_pos, nh, nkv, hd, vd, vo, plan, **how)
        check(got, want, 2e-5, f"plan {plan}")
        assert float(got[tok_seq < 0].abs().sum()) == 0.0


def test_attention_keeps_to_what_a_query_sees(ops):
    """Infinities in the values of keys that a query does not see, in its own tile and page, stay out of its output; a row's bits
    do not depend on the rows beside it."""
    nh, nkv, hd, n = 4, 1, 128, 90
    kp, vp, table, _, _ = scatter_pages(4, nkv, hd, [n], torch.float32, seed=1)
    q = torch.randn(n, nh * hd, generator=torch.Generator().manual_seed(2)).to(DEV)
    seq, pos = torch.zeros(n, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV)
    args = (nh, nkv, hd, hd, hd)
    clean = {plan: run_attention(ops, q, kp, vp, table, seq, pos, *args, plan) for plan in ((0, 0), (128, 1))}
    for at in (5, 70):
        page = int(table[0, at // 64])
        dirty = vp.clone()
        dirty[page, 0, at % 64, 3] = math.inf
        for plan, want in clean.items():
            got = run_attention(ops, q, kp, dirty, table, seq, pos, *args, plan)
            assert torch.equal(got[:at], want[:at]) and torch.isinf(got[at:].view(-1, nh, hd)[:, :, 3]).all()
    for plan, want in clean.items():
        for t in (0, 63, 64, 89):
            one = run_attention(ops, q[t:t + 1], kp, vp, table, seq[t:t + 1].clone(), pos[t:t + 1].clone(), *args, plan)
            assert torch.equal(one[0], want[t])


@pytest.mark.parametrize("m", [17, 40, 200, 300])
def test_many_token_product_keeps_every_bit_of_its_operands(ops, m):
    """A row with a single power of two in it passes the weights through unchanged, whichever side it is on: nothing of a
    number's 24 bits is lost on the way to the tensor cores.  A row with a single number in it gives that product to 2^-22: what is
    left out is 2^-24 of it at most, and the sum of the six products is cut, not rounded, to 24 bits: 2^-23 once or twice."""
    n, k = 1100, 1024
    g = torch.Generator(device=DEV).manual_seed(m)
    work = ops.GemmWorkspace(DEV)

    def product(x, w):
        floats = ops.linear_f32_many_scratch_floats(x.shape[0], w.shape[0], k)
        out = torch.empty(x.shape[0], w.shape[0], device=DEV)
        ops.linear_f32_many(x, w, None, out, torch.empty(floats, device=DEV) if floats else None, work)
        return out

    def single(rows):
        x = torch.zeros(rows, k, device=DEV)
        at = torch.randint(0, k, (rows,), generator=g, device=DEV)
        sign = torch.randint(0, 2, (rows,), generator=g, device=DEV) * 2 - 1
        x[torch.arange(rows, device=DEV), at] = torch.ldexp(sign.float(), torch.randint(-20, 21, (rows,), generator=g, device=DEV))
        return x
    w, x = torch.randn(n, k, generator=g, device=DEV), single(m)
    assert torch.equal(product(x, w).double(), x.double() @ w.double().T)
    w, x = single(n), torch.randn(m, k, generator=g, device=DEV)
    assert torch.equal(product(x, w).double(), x.double() @ w.double().T)
    w, x = torch.randn(n, k, generator=g, device=DEV), single(m) * torch.randn(m, 1, generator=g, device=DEV)
    want = x.double() @ w.double().T
    assert ((product(x, w) - want).abs() <= 2.0 ** -22 * want.abs()).all()
    assert int(work.status.item()) == 0


@pytest.mark.parametrize("m,n", [(40, 1024), (300, 2048)])
@pytest.mark.parametrize("k", [32, 64, 100, 160, 256, 384, 508, 512, 768])
def test_many_token_product_is_as_near_as_the_chain(ops, m, n, k):
    """Over short sums too, where the tensor core's own sums are 32 columns long, the error is no larger than the general kernel's."""
    g = torch.Generator(device=DEV).manual_seed(m + k)
    x, w = torch.randn(m, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV) * 0.02
    floats = ops.linear_f32_many_scratch_floats(m, n, k)
    out, general, work = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV), ops.GemmWorkspace(DEV)
    ops.linear_f32_many(x, w, None, out, torch.empty(floats, device=DEV) if floats else None, work)
    ops.linear_simt(x, w, None, general)
    want = x.double() @ w.double().T
    assert (out - want).norm() <= (general - want).norm() and int(work.status.item()) == 0


@pytest.mark.parametrize("scale_x,scale_w", [(2.0 ** -118, 2.0 ** 10), (2.0 ** -126, 2.0 ** 20), (2.0 ** 100, 2.0 ** -118),
                                             (2.0 ** -80, 2.0 ** -60), (2.0 ** -105, 2.0 ** 60)])
def test_many_token_product_of_tiny_numbers(ops, scale_x, scale_w):
    """Numbers whose last bits lie below the smallest that their parts can be, and sums below float's normal range: as near to
    64-bit sums as a 32-bit sum may be (2^-149 a term, a float's smallest step, on top)."""
    m, n, k = 40, 1100, 1024
    g = torch.Generator(device=DEV).manual_seed(7)
    x, w = torch.randn(m, k, generator=g, device=DEV) * scale_x, torch.randn(n, k, generator=g, device=DEV) * scale_w
    floats = ops.linear_f32_many_scratch_floats(m, n, k)
    out = torch.empty(m, n, device=DEV)
    ops.linear_f32_many(x, w, None, out, torch.empty(floats, device=DEV) if floats else None, ops.GemmWorkspace(DEV))
    assert ((out - x.double() @ w.double().T).abs() <= bound(x, w) + (k + 4) * 2.0 ** -149).all()


def test_a_model_whose_products_are_large(tmp_path):
    """A float32 model whose matrices go to the kernels of this file (2^20 weights and more): a whole prompt, portions of up to 16
    tokens, of more, and token by token, against a float64 statement of the model.  14 products, each as near as 2^-20 in the
    2-norm (measured: 5e-7), and their sum is far above what attention, norms and activations add."""
    from plain_torch import TorchQwen3
    from nncpu_b200 import Engine, Model
    from nncpu_b200.config import config_from_dict
    from nncpu_b200.weights import write_model_folder
    cfg = config_from_dict(dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=2, hidden_size=1024, num_attention_heads=8,
                                num_key_value_heads=2, head_dim=128, intermediate_size=1536, vocab_size=1100, rope_theta=1e6,
                                rms_norm_eps=1e-6, tie_word_embeddings=False, attention_bias=True, max_position_embeddings=4096))
    folder = write_model_folder(tmp_path / "m", cfg, 3, torch.float32)
    toks = torch.randint(0, 1100, (150,), generator=torch.Generator().manual_seed(1)).tolist()
    want = torch.from_numpy(TorchQwen3(folder).logits(toks))
    model = Model.load(folder, dtype="float32", device=DEV)

    def through(cuts):
        engine = Engine(model, max_tokens=256, n_slots=1, max_seq_len=256)
        slot, rows = engine.alloc_slot(), []
        for a, b in zip(cuts, cuts[1:]):
            rows.append(engine.step([slot], [toks[a:b]], [list(range(b - a))]).double().cpu())
        return torch.cat(rows)
    for cuts in ([0, 150], [0, 16, 32, 35, 51, 60, 150], [0, 17, 57, 120, 150], [0, 100] + list(range(101, 151))):
        got = through(cuts)
        assert float((got - want).norm() / want.norm()) <= 14 * 2.0 ** -20, cuts


def test_attention_of_more_tokens_than_a_grid_is_high(ops):
    """Beyond 65 535 decode rows, and beyond 65 535 tiles of query rows (32 query heads on one key/value head: a tile a token)."""
    n = 66001
    g = torch.Generator(device=DEV).manual_seed(3)
    kp, vp = (torch.randn(n, 1, 64, 4, generator=g, device=DEV) for _ in range(2))
    table = torch.randperm(n, generator=g, device=DEV).to(torch.int32).view(n, 1)
    seq = torch.arange(n, dtype=torch.int32, device=DEV)
    pos = torch.randint(0, 64, (n,), generator=g, device=DEV).to(torch.int32)
    q = torch.randn(n, 2 * 4, generator=g, device=DEV)
    want = torch.empty(n, 2 * 4, device=DEV)
    ops.attention(q, kp, vp, table, seq, pos, want, 2, 1, 4, 0.5)
    for plan in ((128, 1), (128, 3)):
        check(run_attention(ops, q, kp, vp, table, seq, pos, 2, 1, 4, 4, 4, plan), want, 2e-5, f"decode rows, plan {plan}")
    pages = (n + 63) // 64
    table = torch.randperm(pages, generator=g, device=DEV).to(torch.int32).view(1, pages)
    seq, pos = torch.zeros(n, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV)
    q = torch.randn(n, 32 * 4, generator=g, device=DEV)
    want = torch.empty(n, 32 * 4, device=DEV)
    ops.attention(q, kp, vp, table, seq, pos, want, 32, 1, 4, 0.5, 70)
    check(run_attention(ops, q, kp, vp, table, seq, pos, 32, 1, 4, 4, 4, (0, 0), window=70), want, 2e-5, "prompt")


def test_sequences_of_a_tile_have_blocks_of_their_own(ops):
    """However many blocks a tile of query rows has for the sequences in it (one, fewer than there are, one for each, more): the same
    bits, padding between them included."""
    nh, nkv, hd = 4, 2, 32
    seqs = [700, 130, 64, 1, 65, 300, 90]
    kp, vp, table, _, _ = scatter_pages(32, nkv, hd, seqs, torch.float32, seed=5)
    tok = [(0, 699), (1, 128), (1, 129), (2, 63), (3, 0), (-1, 9), (4, 64), (5, 299), (6, 88), (6, 89)] + [(5, p) for p in range(40)]
    seq, pos = (torch.tensor([t[i] for t in tok], dtype=torch.int32, device=DEV) for i in (0, 1))
    q = torch.randn(len(tok), nh * hd, generator=torch.Generator().manual_seed(6)).to(DEV)
    want = torch.empty(len(tok), nh * hd, device=DEV)
    ops.attention(q, kp, vp, table, seq, pos, want, nh, nkv, hd, 1 / math.sqrt(hd))
    outs = [run_attention(ops, q, kp, vp, table, seq, pos, nh, nkv, hd, hd, hd, (0, 0), n_seqs=n) for n in (0, 1, 2, 7, 40)]
    check(outs[0], want, 2e-5, "tiles")
    assert all(torch.equal(o, outs[0]) for o in outs[1:])


def test_a_rows_stretches_follow_from_its_own_position(ops):
    """The bits of a token are the same whatever the longest sequence of the step may be and whichever rows stand beside it, in
    decode steps and short portions of up to 64 tokens: 128 keys a stretch up to 4 096, 256 up to 8 192."""
    nh, nkv, hd = 4, 1, 64
    seqs = [700, 4096, 4097, 5000, 90]
    kp, vp, table, _, _ = scatter_pages(260, nkv, hd, seqs, torch.float32, seed=8)
    seq = torch.arange(5, dtype=torch.int32, device=DEV)
    pos = torch.tensor([n - 1 for n in seqs], dtype=torch.int32, device=DEV)
    q = torch.randn(5, nh * hd, generator=torch.Generator().manual_seed(9)).to(DEV)
    want = torch.empty(5, nh * hd, device=DEV)
    ops.attention(q, kp, vp, table, seq, pos, want, nh, nkv, hd, 1 / math.sqrt(hd))
    args = (nh, nkv, hd, hd, hd)
    whole = run_attention(ops, q, kp, vp, table, seq, pos, *args, ops.attention_f32_plan(5, True, 5000, 5))
    check(whole, want, 2e-5, "token by token")
    assert torch.equal(whole, run_attention(ops, q, kp, vp, table, seq, pos, *args, ops.attention_f32_plan(5, True, 40960, 5)))
    for t, n in enumerate(seqs):
        for longest in (n, 5000, 40960):
            plan = ops.attention_f32_plan(1, False, longest)
            one = run_attention(ops, q[t:t + 1], kp, vp, table, seq[t:t + 1].clone(), pos[t:t + 1].clone(), *args, plan)
            assert torch.equal(one[0], whole[t]), (n, longest)
