"""Element-wise kernels in whole words: sizes around a CTA's share of a row, against the same operations of torch (GPU)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("tokens,top,width", [(1, 1, 4), (8, 4, 4096), (3, 8, 1020), (5, 9, 1024), (2, 3, 1030), (300, 2, 2052)])
@pytest.mark.parametrize("always,out_type", [(None, torch.float32), (torch.bfloat16, torch.float32), (torch.float32, torch.bfloat16)])
def test_expert_combine(tokens, top, width, always, out_type):
    """Up to eight choices in words, more or odd widths one by one: sums of `top` terms, 2^-24 each, then the output's rounding."""
    from lucciola_b200 import ops
    torch.manual_seed(1)
    places = tokens * top + 7
    y, w = torch.randn(places, width, device=DEV), torch.rand(tokens, top, device=DEV)
    at = torch.randperm(places, device=DEV)[:tokens * top].to(torch.int32)
    a = torch.randn(tokens, width, device=DEV).to(always) if always else None
    out = torch.empty(tokens, width, dtype=out_type, device=DEV)
    ops.expert_combine(out, y, w, at, stream(), always=a)
    want = (w.double()[..., None] * y[at.long()].view(tokens, top, width).double()).sum(1) + (a.double() if always else 0.0)
    assert (out.double() - want).abs().max() <= (2e-6 if out_type == torch.float32 else 8e-3) * want.abs().max()


@pytest.mark.parametrize("tokens,hidden,scale", [(1, 4, 1.0), (8, 2048, 1.0), (9, 1028, 2.0), (300, 4096, 1.0), (3, 66, 0.5)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embedding_rows(tokens, hidden, scale, dtype):
    """Rows of the table times a power of two: exact; ids outside it read row 0."""
    from lucciola_b200 import ops
    table = torch.randn(50, hidden, device=DEV).to(dtype)
    ids = torch.randint(0, 50, (tokens,), dtype=torch.int32, device=DEV)
    ids[-1] = 77
    out = torch.empty(tokens, hidden, device=DEV)
    ops.embedding(out, ids, table, stream(), scale=scale)
    want = table.float()[torch.where(ids < 50, ids, 0).long()] * scale
    assert torch.equal(out, want)


@pytest.mark.parametrize("nq,nkv,d", [(1, 1, 64), (3, 1, 64), (5, 2, 128), (32, 8, 128), (2, 1, 256), (7, 3, 256)])
@pytest.mark.parametrize("tokens", [1, 9, 700])
@pytest.mark.parametrize("norm,rotate,pages,pad", [("qk", True, True, 0), ("k", True, False, 0), ("q", False, True, 8), ("", True, True, 0), ("qk", True, True, 4),
                                                   ("qk", True, False, 2)])
def test_rope_rows(nq, nkv, d, tokens, norm, rotate, pages, pad):
    """Heads of whole 16-byte words (pad 0 and 8) and rows that are not: the result's rounding, 2^-9 of each, behind 32-bit sums."""
    from lucciola_b200 import ops
    torch.manual_seed(tokens + nq)
    a, b, ps = nq * d, (nq + nkv) * d, 16
    qkv = torch.randn(tokens, b + nkv * d + pad, device=DEV).bfloat16()
    weight = lambda on: 1 + 0.2 * torch.randn(d, device=DEV) if on else None
    qw, kw = weight("q" in norm), weight("k" in norm)
    inv = 1e4 ** (-torch.arange(0, d, 2, device=DEV, dtype=torch.float32) / d) if rotate else None
    pos = torch.arange(tokens, device=DEV, dtype=torch.int32) * 3 + 5
    seq = torch.arange(tokens, device=DEV, dtype=torch.int32) % 3
    table = torch.randperm(3 * (tokens * 3 // ps + 2), device=DEV).to(torch.int32).view(3, -1).contiguous()
    q_out = torch.empty(tokens, nq, d, device=DEV, dtype=torch.bfloat16)
    shape = (table.numel(), nkv, ps, d) if pages else (tokens, nkv, d)
    k_to, v_to = torch.full(shape, 9.0, device=DEV).bfloat16(), torch.full(shape, 9.0, device=DEV).bfloat16()
    into = dict(k_cache=k_to, v_cache=v_to, token_seq=seq, block_table=table, page_size=ps) if pages else dict(k_out=k_to, v_out=v_to)
    ops.rope_kv(qkv[:, :a], qkv[:, a:b], qkv[:, b:b + nkv * d], q_out, pos, nq, nkv, d, 1e-6, stream(), q_norm_w=qw, k_norm_w=kw,
                inv_freq=inv, rot_dim=d if rotate else 0, **into)

    def plain(x, w):
        x = x.double()
        if w is not None:
            x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w.double()
        if inv is not None:
            at = (pos.float()[:, None] * inv).double()[:, None]
            lo, hi = x[..., :d // 2], x[..., d // 2:]
            x = torch.cat([lo * at.cos() - hi * at.sin(), lo * at.sin() + hi * at.cos()], -1)
        return x

    def near(got, want):
        return bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all())

    assert near(q_out, plain(qkv[:, :a].reshape(tokens, nq, d), qw))
    if pages:
        page = table[seq.long(), (pos // ps).long()].long()
        k_got, v_got = k_to[page, :, (pos % ps).long()], v_to[page, :, (pos % ps).long()]
        assert (v_to != 9).any(-1).sum() == tokens * nkv                              # no other slot was written
    else:
        k_got, v_got = k_to, v_to
    assert near(k_got, plain(qkv[:, a:b].reshape(tokens, nkv, d), kw))
    assert torch.equal(v_got, qkv[:, b:b + nkv * d].reshape(tokens, nkv, d))


@pytest.mark.parametrize("M,N,K", [(1, 1, 8), (8, 16, 4096), (7, 128, 2048), (9, 33, 5000), (16, 64, 2056), (3, 16, 8192), (16, 128, 16384), (16, 128, 16392)])
@pytest.mark.parametrize("out_type,post", [(torch.float32, None), (torch.bfloat16, None), (torch.float32, "cap")])
def test_product_of_few_features(M, N, K, out_type, post):
    """K products of bfloat16 values summed in 32 bits; each feature is a CTA's, so the sizes around its words and tokens matter;
    from 16385 places on the pipeline for few tokens takes them, in chains no longer than the bound."""
    from lucciola_b200 import ops
    torch.manual_seed(M)
    x, w = torch.randn(M, K + 8, device=DEV).bfloat16()[:, 8:], torch.randn(N, K, device=DEV).bfloat16()
    y = torch.full((M, N + 1), 7.0, dtype=out_type, device=DEV)
    ops.gemm_tcgen05(y[:, :N], x, w, stream(), post=post, post_c=5.0)
    terms = x.double()[:, None] * w.double()
    want = terms.sum(-1)
    if post:
        want = 5.0 * torch.tanh(want / 5.0)
    bound = (K / 256 + 13) * 2.0 ** -24 * terms.abs().sum(-1) + (2.0 ** -8 * want.abs() if out_type == torch.bfloat16 else 0) + 1e-6 * (post is not None)
    assert ((y[:, :N].double() - want).abs() <= bound).all() and (y[:, N] == 7).all()


@pytest.mark.parametrize("T,channels,n", [(1, 4, 4), (5, 260, 128), (64, 6144, 124), (3, 512, 300)])
def test_conv_step_rounds_on_the_way(T, channels, n):
    """The convolution's step with columns to round: both as the launches that do one of them, to the bit."""
    from types import SimpleNamespace
    from lucciola_b200 import ops
    torch.manual_seed(T)
    x, w = torch.randn(T, channels + n + 4, device=DEV), torch.randn(4, channels, device=DEV)
    state = torch.randn(T + 1, 3, channels, device=DEV)
    step = SimpleNamespace(max_q_len=1, q_lens=[1] * T, num_seqs=T, state_slots=torch.arange(T, 0, -1, dtype=torch.int32, device=DEV))
    want, state2 = torch.empty(T, channels, device=DEV), state.clone()
    assert ops.short_conv_step(want, x[:, :channels], w, None, state, step, stream())
    first, plain = (torch.empty(T, n, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    ops.round_cols(plain, x[:, channels:channels + n], stream())
    got = torch.empty_like(want)
    assert ops.short_conv_step(got, x[:, :channels], w, None, state2, step, stream(), rounded=(first, x[:, channels:channels + n]))
    assert torch.equal(got, want) and torch.equal(state2, state) and torch.equal(first, plain)


@pytest.mark.parametrize("heads,M,N,K", [(32, 64, 128, 512), (32, 33, 512, 128), (3, 17, 33, 40), (70, 64, 128, 512), (1, 1, 2, 8), (5, 48, 34, 264)])
@pytest.mark.parametrize("gates", [0, 1, 2])
def test_heads_of_few_rows(heads, M, N, K, gates):
    """The tokens' shares by the number of heads, odd widths (no pairs of stores), rows of longer heads: K products in 32 bits, then bfloat16."""
    from lucciola_b200 import ops
    torch.manual_seed(M + N)
    x = torch.randn(M, heads, K + 8, device=DEV).bfloat16()[:, :, 8:]
    w = torch.randn(heads, N, K, device=DEV).bfloat16()
    gate = torch.randn(M, heads * (N if gates == 2 else 1), device=DEV) if gates else None
    y = torch.full((M, heads, N + 1), 9.0, device=DEV).bfloat16()
    ops.gemm_heads(y[:, :, :N], x, w, stream(), gate=gate)
    xd, wd = x.double(), w.double()
    want, size = torch.einsum("mhk,hnk->mhn", xd, wd), torch.einsum("mhk,hnk->mhn", xd.abs(), wd.abs())
    if gates:
        g = torch.sigmoid(gate.double()).view(M, heads, -1)
        want, size = want * g, size * g
    assert ((y[:, :, :N].double() - want).abs() <= 2.0 ** -8 * want.abs() + (K / 8 + 4) * 2.0 ** -24 * size).all() and (y[:, :, N] == 9).all()
