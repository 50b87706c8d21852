"""Long portions of the linear recurrences, 64 tokens at a time, and steps of single tokens, against the plain recurrence in 64 bits and against the
token-by-token kernels: every kind, portions around the edges of a block, a chunk and several, sizes that fill no tile, inputs
that are column ranges, portions beside single tokens, and scratch for fewer chunks than there are (GPU)."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def step_of(lens, slots):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    return SimpleNamespace(num_seqs=len(lens), cu_tokens=i32(cu), state_slots=i32(slots), q_lens=list(lens), max_q_len=max(lens))


def columns(x):
    """The same values as a column range of a wider matrix whose rows start on no 16-byte boundary."""
    return torch.cat([torch.zeros(x.shape[0], 3, device=DEV), x, torch.zeros(x.shape[0], 2, device=DEV)], dim=1)[:, 3:3 + x.shape[1]]


def operands(kind, T, heads, groups, dim, vdim):
    rnd = lambda *s: torch.randn(*s, device=DEV)
    o = dict(v=rnd(T, heads * vdim))
    if kind == "fixed":
        o.update(q=rnd(T, heads * dim), k=rnd(T, heads * dim), decay=torch.tensor([0.999, 0.5, 1.0, 0.97, 0.9, 0.0][:heads], device=DEV))
    elif kind == "hgrn2":
        o.update(q=rnd(T, heads * dim), k=2 * rnd(T, heads * dim), bias=rnd(heads * dim), lower=torch.rand(heads * dim, device=DEV))
        o["lower"][::3] = 0.0
        o["bias"][::5] = -30.0                                    # gates of next to nothing: products that leave the range of 32 bits
    else:
        o.update(q=rnd(T, groups * dim), k=rnd(T, groups * dim), a=rnd(T, heads), b=rnd(T, heads), A_log=torch.rand(heads, device=DEV) * 2,
                 dt_bias=rnd(heads) - 2)
        if kind == "ssm":
            o.update(D=rnd(heads), b=None)
        if kind == "channels":
            o.update(a=3 * rnd(T, heads * dim), dt_bias=rnd(heads * dim) - 2)
    return o


def through_ops(kind, o, state, step, heads, groups, dim, vdim, by_shape, shifted=True):
    """`shifted`: the operands that may be column ranges start on no 16-byte boundary."""
    from lucciola_b200 import ops
    s = torch.cuda.current_stream().cuda_stream
    T = o["v"].shape[0]
    out = torch.full((T, heads * vdim), float("nan"), device=DEV)
    n, m = heads * dim, heads * vdim
    at = columns if shifted else (lambda x: x)
    if kind == "fixed":
        pre = at(torch.cat([o["q"], o["k"], o["v"]], dim=1))
        ops.decay_recurrence(pre, 0, n, 2 * n, o["decay"], state, out, step, heads, dim, vdim, s, by_shape=by_shape)
    elif kind == "hgrn2":
        pre = torch.cat([o["q"], o["k"], o["v"]], dim=1)          # whole rows: their alignment follows from the sizes
        ops.gated_recurrence(pre, 0, n, 2 * n, o["bias"], o["lower"], state, out, step, heads, dim, vdim, s, by_shape=by_shape)
    else:
        delta = kind != "ssm"
        ops.state_recurrence(at(o["q"]), o["k"], at(o["v"]), at(o["a"].clone()), o["b"], o["A_log"], o["dt_bias"], o.get("D"), state, out, step, heads,
                             groups, dim, vdim, s, delta=delta, unit_norm=delta, q_scale=dim ** -0.5 if delta else 1.0, rows_decay=kind == "channels",
                             by_shape=by_shape)
    return out


def plain(kind, o, state, step, heads, groups, dim, vdim):
    d = {k: (t.double() if t is not None else None) for k, t in o.items()}
    T, silu, soft = d["v"].shape[0], torch.nn.functional.silu, torch.nn.functional.softplus
    v = d["v"].view(T, heads, 1, vdim)
    q, k = (d[x].view(T, -1, dim) for x in "qk")
    g, w = torch.ones(T, heads, 1, 1, dtype=torch.float64, device=DEV), torch.ones(T, heads, 1, dtype=torch.float64, device=DEV)
    if kind == "fixed":
        q, k, v = silu(q), silu(k), silu(v)
        g = g * d["decay"][:, None, None]
    elif kind == "hgrn2":
        low = d["lower"].view(heads, dim)
        q, f = silu(q), low + (1 - low) * torch.sigmoid(k + d["bias"].view(heads, dim))
        g, k = f[..., None], 1 - f
    else:
        x = soft(d["a"] + d["dt_bias"])
        if kind == "channels":
            g = torch.exp(-torch.exp(d["A_log"])[:, None] * x.view(T, heads, dim))[..., None]
        else:
            g = torch.exp(-torch.exp(d["A_log"]) * x)[..., None, None]
        if kind == "ssm":
            w = x[..., None]
        else:
            q, k = (y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6) for y in (q, k))
            q, w = q * dim ** -0.5, torch.sigmoid(d["b"])[..., None]
        q, k = (y.repeat_interleave(heads // groups, 1) for y in (q, k))
    out, S, at = [], state.double().clone(), 0
    for i, n in enumerate(step.q_lens):
        slot = int(step.state_slots[i])
        for t in range(at, at + n):
            X = g[t] * S[slot]
            seen = (X * k[t][..., None]).sum(1) if kind in ("delta", "channels") else 0.0
            X = X + k[t][..., None] * (w[t] * (v[t, :, 0] - seen))[:, None]
            S[slot] = X
            y = (X * q[t][..., None]).sum(1)
            out.append(y + d["D"][:, None] * v[t, :, 0] if kind == "ssm" else y)
        at += n
    return torch.stack(out).reshape(T, -1), S


@pytest.fixture(autouse=True)
def from_32_tokens(monkeypatch):
    """Whatever it costs: the chunked form for every portion that it may take."""
    from lucciola_b200 import ops
    monkeypatch.setattr(ops, "chunk_portions", lambda kind, step, *sizes: ([i for i, n in enumerate(step.q_lens) if n >= 32], 32))


@pytest.mark.parametrize("heads,groups,dim,vdim,lens", [
    (2, 1, 128, 128, [64]), (3, 3, 128, 128, [63, 65]), (2, 2, 64, 64, [32, 200]), (4, 2, 20, 40, [33, 1, 129]), (2, 1, 72, 33, [1, 2, 47, 130, 31]),
    (1, 1, 128, 8, [256]), (6, 3, 100, 72, [300]), (5, 5, 8, 6, [80])])
@pytest.mark.parametrize("kind", ["fixed", "ssm", "hgrn2", "delta", "channels"])
@pytest.mark.parametrize("shifted", [False, True])
def test_long_portions(kind, heads, groups, dim, vdim, lens, shifted):
    """Outputs and states within 1e-5 of their largest value: a few hundred terms of 2^-24 relative error each, as for the
    kernels that walk token by token; rows of the state that belong to nobody stay as they are."""
    torch.manual_seed(3)
    o = operands(kind, sum(lens), heads, groups, dim, vdim)
    slots = list(range(len(lens), 0, -1))
    step = step_of(lens, slots)
    state = 0.3 * torch.randn(len(lens) + 2, heads, dim, vdim, device=DEV)
    state[0] = state[-1] = float("nan")
    want, S = plain(kind, o, state, step, heads, groups, dim, vdim)
    for by_shape in (True, False):
        got_state = state.clone()
        got = through_ops(kind, o, got_state, step, heads, groups, dim, vdim, by_shape, shifted)
        assert (got.double() - want).abs().max() <= 1e-5 * want.abs().max(), by_shape
        live = got_state[1:-1].double()
        assert (live - S[1:-1]).abs().max() <= 1e-5 * S[1:-1].abs().max(), by_shape
        assert torch.isnan(got_state[0]).all() and torch.isnan(got_state[-1]).all()


@pytest.mark.parametrize("heads,dim,vdim", [(16, 128, 128), (32, 128, 128), (16, 128, 120), (32, 100, 120), (16, 64, 128), (32, 64, 128), (32, 40, 120)])
@pytest.mark.parametrize("kind", ["delta", "channels"])
@pytest.mark.parametrize("shifted", [False, True])
def test_walks_of_wider_columns(kind, heads, dim, vdim, shifted):
    """The walk over the chunks takes 32 value columns a CTA where that makes 100 CTAs (here 32 heads), else 16 (here 16 heads), else 8
    (test_long_portions); the bounds of test_long_portions."""
    torch.manual_seed(10)
    lens = [90, 70]
    o = operands(kind, sum(lens), heads, heads // 2, dim, vdim)
    for one in range(2):                                          # a sequence a step, so that its heads alone choose the width
        n = lens[one]
        mine = {k: (x[:n] if x is not None and x.shape[0] == sum(lens) else x) for k, x in o.items()}
        step = step_of([n], [1])
        state = 0.3 * torch.randn(2, heads, dim, vdim, device=DEV)
        want, S = plain(kind, mine, state, step, heads, heads // 2, dim, vdim)
        got = through_ops(kind, mine, state, step, heads, heads // 2, dim, vdim, True, shifted)
        assert (got.double() - want).abs().max() <= 1e-5 * want.abs().max()
        assert (state[1].double() - S[1]).abs().max() <= 1e-5 * S[1].abs().max()


@pytest.mark.parametrize("heads,groups,dim,vdim,lens", [(4, 2, 128, 128, [600]), (3, 3, 64, 128, [250, 90]), (4, 1, 128, 64, [40, 333])])
@pytest.mark.parametrize("kind", ["fixed", "ssm", "hgrn2", "delta", "channels"])
def test_as_exact_as_token_by_token(kind, heads, groups, dim, vdim, lens):
    """Outputs (before any norm) and states against 64 bits: no further off than those of the kernels that walk token by token, in
    the 2-norm over some 1e5 values, for operands as the layers have them (rates and steps as the designs initialise them, rows behind
    a convolution's silu).  Measured ratios over the layers' sizes 0.2 to 0.98, a tenth for another seed; operands or sums of
    fewer bits than 24 showed 1.2 to 6."""
    torch.manual_seed(8)
    T, silu = sum(lens), torch.nn.functional.silu
    o = operands(kind, T, heads, groups, dim, vdim)
    if kind == "fixed":
        o["decay"] = 1 - 2.0 ** -torch.linspace(3, 11, heads, device=DEV)
    elif kind == "hgrn2":
        o.update(k=0.9 * torch.randn(T, heads * dim, device=DEV), bias=0.02 * torch.randn(heads * dim, device=DEV), lower=torch.rand(heads * dim, device=DEV))
    else:
        dt = torch.exp(torch.rand(o["dt_bias"].shape, device=DEV) * 4.6 - 6.9)
        o.update(q=silu(o["q"]), k=silu(o["k"]), v=silu(o["v"]), A_log=torch.log(1 + 15 * torch.rand(heads, device=DEV)), dt_bias=dt + torch.log(-torch.expm1(-dt)),
                 a=0.5 * torch.randn(o["a"].shape, device=DEV))
    step = step_of(lens, list(range(len(lens))))
    state = 0.3 * torch.randn(len(lens), heads, dim, vdim, device=DEV)
    want, S = plain(kind, o, state, step, heads, groups, dim, vdim)
    off = {}
    for by_shape in (True, False):
        got_state = state.clone()
        got = through_ops(kind, o, got_state, step, heads, groups, dim, vdim, by_shape)
        off[by_shape] = torch.stack([(got.double() - want).norm() / want.norm(), (got_state.double() - S).norm() / S.norm()])
    assert (off[True] <= 1.1 * off[False]).all(), off


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("where,token,column", [("v", 37, 5), ("v", 32, 9), ("v", 70 + 47, 70), ("k", 40, 7), ("k", 70 + 64, 3), ("q", 50, 1), ("a", 41, 0), ("b", 43, 1)])
@pytest.mark.parametrize("kind", ["fixed", "ssm", "hgrn2", "delta", "channels"])
def test_what_is_not_finite_stays_with_its_tokens(kind, where, token, column, bad):
    """One infinity or NaN in the first or second of three portions: outputs and states are finite exactly where the kernels that
    walk token by token have them finite, and there as close to 64 bits as ever."""
    heads, groups, dim, vdim, lens = 2, 2, 64, 72, [70, 130, 40]
    torch.manual_seed(9)
    o = operands(kind, sum(lens), heads, groups, dim, vdim)
    if kind == "fixed":
        o["decay"] = torch.tensor([0.97, 0.9], device=DEV)
    if o.get(where) is None:
        pytest.skip("this recurrence has no such operand")
    step = step_of(lens, [2, 0, 1])
    state = 0.3 * torch.randn(4, heads, dim, vdim, device=DEV)
    o[where][token, column] = bad
    want, S = plain(kind, o, state, step, heads, groups, dim, vdim)
    got_state, walked_state = state.clone(), state.clone()
    got = through_ops(kind, o, got_state, step, heads, groups, dim, vdim, True)
    walked = through_ops(kind, o, walked_state, step, heads, groups, dim, vdim, False)
    for x, y, z in ((got, walked, want), (got_state[:3], walked_state[:3], S[:3])):
        assert torch.equal(torch.isfinite(x), torch.isfinite(y))
        same = torch.isfinite(y) & torch.isfinite(z)
        assert (x.double() - z).abs()[same].max() <= 1e-5 * z[same].abs().max()
    before = torch.arange(sum(lens), device=DEV) < token
    assert torch.isfinite(got[before]).all() and torch.isfinite(got[sum(lens[:2]):]).all()


@pytest.mark.parametrize("seqs,heads,groups,dim,vdim", [(1, 2, 1, 128, 128), (3, 4, 2, 64, 64), (80, 4, 4, 128, 128), (5, 64, 2, 128, 64), (40, 8, 4, 72, 68), (2, 3, 3, 65, 260),
                                                        (150, 2, 1, 100, 132), (7, 2, 1, 33, 132), (9, 3, 3, 64, 60)])
@pytest.mark.parametrize("kind", ["fixed", "ssm", "hgrn2", "delta", "channels"])
def test_single_tokens(kind, seqs, heads, groups, dim, vdim):
    """One token a sequence, in every width of CTA: the bounds of test_long_portions, and close to the kernels that walk tokens."""
    from lucciola_b200 import ops
    torch.manual_seed(5)
    o = operands(kind, seqs, heads, groups, dim, vdim)
    if kind == "fixed":
        o["decay"] = torch.rand(heads, device=DEV)
    step = step_of([1] * seqs, list(range(seqs, 0, -1)))
    state = 0.3 * torch.randn(seqs + 2, heads, dim, vdim, device=DEV)
    state[0] = state[-1] = float("nan")
    assert ops.single_tokens(step, dim, vdim, state) == (dim >= 64 and vdim >= 64)      # smaller states are walked either way
    want, S = plain(kind, o, state, step, heads, groups, dim, vdim)
    for by_shape in (True, False):
        got_state = state.clone()
        got = through_ops(kind, o, got_state, step, heads, groups, dim, vdim, by_shape)
        assert (got.double() - want).abs().max() <= 1e-5 * want.abs().max(), by_shape
        assert (got_state[1:-1].double() - S[1:-1]).abs().max() <= 1e-5 * S[1:-1].abs().max(), by_shape
        assert torch.isnan(got_state[0]).all() and torch.isnan(got_state[-1]).all()


@pytest.mark.parametrize("kind", ["fixed", "delta", "channels"])
def test_scratch_for_fewer_chunks_and_more_sequences_than_a_launch(kind, monkeypatch):
    """The chunks of three sequences in turns of two, the same bits as in one; more than 64 long sequences in a step."""
    from lucciola_b200 import ops
    heads, dim, vdim, lens = 2, 64, 40, [150, 64, 90]
    torch.manual_seed(4)
    o = operands(kind, sum(lens), heads, heads, dim, vdim)
    state = torch.randn(5, heads, dim, vdim, device=DEV)
    step = step_of(lens, [2, 0, 3])
    whole_state = state.clone()
    whole = through_ops(kind, o, whole_state, step, heads, heads, dim, vdim, True)
    one = ops._chunk_floats(ops._CHUNK_KINDS[kind], heads, dim, vdim)
    monkeypatch.setattr(ops, "CHUNK_SCRATCH", 2 * one + 1)
    turned = through_ops(kind, o, state, step, heads, heads, dim, vdim, True)
    assert torch.equal(turned, whole) and torch.equal(state, whole_state)
    lens = [32 + i % 3 for i in range(70)]
    o = operands(kind, sum(lens), heads, heads, dim, vdim)
    step = step_of(lens, list(range(70)))
    state = torch.randn(71, heads, dim, vdim, device=DEV)
    want, S = plain(kind, o, state, step, heads, heads, dim, vdim)
    got = through_ops(kind, o, state, step, heads, heads, dim, vdim, True)
    assert (got.double() - want).abs().max() <= 1e-5 * want.abs().max() and (state.double() - S).abs().max() <= 1e-5 * S.abs().max()


def test_scratch_where_memory_is_scant(monkeypatch):
    """Where the allocator has no room for all chunks at once they are worked off in more turns, the same bits; and where there is none for
    those either, the call fails as any other does that finds no memory."""
    from lucciola_b200 import ops
    heads, dim, vdim, T = 32, 128, 128, 1900
    torch.manual_seed(12)
    o = operands("hgrn2", T, heads, heads, dim, vdim)
    state, step = torch.randn(1, heads, dim, vdim, device=DEV), step_of([T], [0])
    one = 4 * ops._chunk_floats(ops._CHUNK_KINDS["hgrn2"], heads, dim, vdim)
    assert 4 * ops.CHUNK_SCRATCH_SCANT < 30 * one <= 4 * ops.CHUNK_SCRATCH
    whole_state = state.clone()
    whole = through_ops("hgrn2", o, whole_state, step, heads, heads, dim, vdim, True)
    total = torch.cuda.get_device_properties(0).total_memory
    rows = 4 * T * heads * (2 * dim + 2 * vdim)            # through_ops lays q, k, v side by side, and the outputs
    real, turns = ops._call, []

    def call(name, *args):
        if name == "lb_chunk_recurrence":
            turns.append(-(-30 // args[-2]))               # of as many chunks as the scratch holds
        real(name, *args)
    monkeypatch.setattr(ops, "_call", call)
    try:
        for room, fits in ((160 << 20, True), (40 << 20, False)):
            got_state = state.clone()
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
            torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + rows + room) / total)
            if fits:
                got = through_ops("hgrn2", o, got_state, step, heads, heads, dim, vdim, True)
                assert turns == [2] and torch.equal(got, whole) and torch.equal(got_state, whole_state)
            else:
                with pytest.raises(torch.OutOfMemoryError):
                    through_ops("hgrn2", o, got_state, step, heads, heads, dim, vdim, True)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


@pytest.mark.parametrize("channels,lens", [(8192, [1]), (260, [1] * 9), (4096, [700, 1, 2, 3, 4, 5, 333]), (4096, [1205, 1, 2, 3, 4, 9, 333]), (1028, [9, 200]), (64, [3000]), (2048, [5, 4, 1, 1, 90])])
@pytest.mark.parametrize("bias", [False, True])
def test_short_convolution_of_several_tokens_a_thread(channels, lens, bias):
    """Portions that start and end anywhere in a thread's two, four or eight tokens, and steps of single tokens with the state in the same launch:
    the very sums of the token-a-thread kernel (any taps and alignment), so the same bits."""
    from lucciola_b200 import ops
    torch.manual_seed(6)
    T, s = sum(lens), torch.cuda.current_stream().cuda_stream
    x = torch.randn(T, channels + 4, device=DEV)[:, 4:]
    w, b = torch.randn(4, channels, device=DEV), torch.randn(channels, device=DEV) if bias else None
    state = torch.randn(len(lens) + 1, 3, channels, device=DEV)
    step = step_of(lens, list(range(len(lens), 0, -1)))
    step.token_seq = torch.tensor([i for i, n in enumerate(lens) for _ in range(n)], dtype=torch.int32, device=DEV)
    odd = torch.cat([torch.zeros(T, 1, device=DEV), x], dim=1)[:, 1:]                      # rows on no 16-byte boundary: four bytes at a time
    want, got, state2 = torch.empty(T, channels, device=DEV), torch.empty(T, channels, device=DEV), state.clone()
    ops.short_conv(want, odd, w, b, state, step, s)
    ops.short_conv_state(state, odd, 4, step, s)
    if ops.short_conv_step(got, x, w, b, state2, step, s):
        assert max(lens) == 1
    else:
        assert max(lens) > 1
        ops.short_conv(got, x, w, b, state2, step, s)
        ops.short_conv_state(state2, x, 4, step, s)
    assert torch.equal(got, want) and torch.equal(state2, state)


@pytest.mark.parametrize("rows,n,groups,planes", [(5, 2048, 16, 1), (3, 2048, 2, 1), (70, 4096, 1, 1), (2, 96, 8, 2), (9, 1040, 2, 3), (4, 8192, 1, 1), (3, 128, 4, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_norms_in_words(rows, n, groups, planes, dtype):
    """Groups around the sizes at which a group takes another number of warps and words a lane, against the formula in 64 bits."""
    from lucciola_b200 import ops
    torch.manual_seed(7)
    s, eps = torch.cuda.current_stream().cuda_stream, 1e-6
    y, gate, w = torch.randn(planes, rows, n, device=DEV), torch.randn(rows, n + 8, device=DEV)[:, 8:], torch.randn(n // groups, device=DEV)
    Y, Z, tol = y.double().sum(0), gate.double(), 3e-6 if dtype == torch.float32 else 8e-3
    parts = lambda z: z / torch.sqrt((z.view(rows, groups, -1) ** 2).mean(-1, keepdim=True) + eps).expand(-1, -1, n // groups).reshape(rows, n)
    for first in (False, True):
        out = torch.empty(rows, n, dtype=dtype, device=DEV)
        ops.gated_group_norm(out, y if planes > 1 else y[0], gate, w, groups, eps, s, gate_first=first, scale=0.5)
        act = torch.nn.functional.silu(Z)
        want = 0.5 * (parts(Y * act) if first else parts(Y) * act) * w.double().repeat(groups)
        assert (out.double() - want).abs().max() <= tol * want.abs().max()
    if groups == 1:
        out = torch.empty(rows, n, dtype=dtype, device=DEV)
        ops.rmsnorm_gated(out, y if planes > 1 else y[0], w, gate, 0.5, eps, s)
        want = 0.5 * parts(Y) * w.double() * torch.sigmoid(Z)
        assert (out.double() - want).abs().max() <= tol * want.abs().max()
