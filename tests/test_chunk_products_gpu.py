"""The chunked recurrences where their products' tiles, rings and CTAs change over: value columns in one tile of 64, of 128 and in several,
more (chunk, head)s than SMs, so that a CTA takes several one behind the other, and a value that is not finite behind the first
tile of columns; against the plain recurrence in 64 bits; and waits that run out (GPU)."""
import ctypes
import time

import pytest
import torch

from test_chunk_recurrence_gpu import DEV, operands, plain, step_of, through_ops

pytestmark = pytest.mark.gpu
KINDS = ["fixed", "ssm", "hgrn2", "delta", "channels"]


@pytest.fixture(autouse=True)
def every_portion(monkeypatch):
    """Whatever it costs: the chunked form for every portion that it may take."""
    from lucciola_b200 import ops
    monkeypatch.setattr(ops, "chunk_portions", lambda kind, step, *sizes: ([i for i, n in enumerate(step.q_lens) if n >= 32], 32))


def gentle(kind, T, heads, groups, dim, vdim):
    o = operands(kind, T, heads, groups, dim, vdim)
    if kind == "fixed":
        o["decay"] = torch.linspace(0.0, 1.0, heads, device=DEV)
    return o


@pytest.mark.parametrize("heads,groups,dim,vdim,lens", [
    (2, 1, 128, 260, [130]), (3, 3, 64, 300, [40, 200]), (2, 2, 128, 65, [64, 63]), (1, 1, 65, 129, [100]),
    (40, 20, 64, 64, [33, 700]), (33, 11, 128, 128, [1, 640]), (20, 20, 128, 136, [570]), (52, 13, 64, 128, [800])])
@pytest.mark.parametrize("kind", KINDS)
def test_tiles_of_columns_and_chunks_behind_one_another(kind, heads, groups, dim, vdim, lens):
    """Within 1e-5 of the largest value, as the kernels that walk token by token: a few hundred terms of 2^-24 relative error each."""
    from lucciola_b200 import ops
    torch.manual_seed(17)
    o = gentle(kind, sum(lens), heads, groups, dim, vdim)
    step = step_of(lens, list(range(len(lens))))
    state = 0.3 * torch.randn(len(lens), heads, dim, vdim, device=DEV)
    want, S = plain(kind, o, state, step, heads, groups, dim, vdim)
    got = through_ops(kind, o, state, step, heads, groups, dim, vdim, True, shifted=False)
    assert (got.double() - want).abs().max() <= 1e-5 * want.abs().max()
    assert (state.double() - S).abs().max() <= 1e-5 * S.abs().max()
    assert ops.device_error() == 0


@pytest.mark.parametrize("column", [3, 127, 128, 259])
@pytest.mark.parametrize("token", [0, 40, 64, 100])
@pytest.mark.parametrize("kind", KINDS)
def test_a_bad_value_in_any_tile_of_columns(kind, token, column):
    """Its column from its token on, and nothing before it or beside it."""
    torch.manual_seed(18)
    lens, heads, dim, vdim = [130], 2, 128, 260
    o = gentle(kind, 130, heads, heads, dim, vdim)
    step = step_of(lens, [0])
    state = 0.3 * torch.randn(1, heads, dim, vdim, device=DEV)
    good = through_ops(kind, o, state.clone(), step, heads, heads, dim, vdim, True, shifted=False)
    o["v"][token, column] = float("nan")
    after = state.clone()
    got = through_ops(kind, o, after, step, heads, heads, dim, vdim, True, shifted=False)
    assert torch.equal(got[:token], good[:token])
    beside = torch.arange(heads * vdim, device=DEV) != column
    assert torch.equal(got[:, beside], good[:, beside])
    assert torch.isnan(got[token:, column]).all() and torch.isnan(after[0, 0, :, column]).all()


@pytest.mark.parametrize("hold,kind,code", [(1, "fixed", 401), (1, "ssm", 401), (1, "hgrn2", 401), (2, "delta", 450), (2, "channels", 450), (4, "delta", 450), (4, "channels", 450)]
                         + [(hold, kind, 410) for hold in (8, 16) for kind in KINDS])
@pytest.mark.parametrize("heads,dim,vdim", [(2, 128, 128), (40, 128, 40), (8, 128, 260), (3, 64, 64)])
def test_a_wait_that_runs_out(hold, kind, code, heads, dim, vdim, monkeypatch):
    """Without the products of K^T U (1), the copies (2) or products (4) of the walk, the copies (8) or products (16) of the outputs, and a limit of
    200 000 cycles, 0.1 ms: the kernel returns, leaves the number of the wait, stores no output and (the walk) no state, with copies in flight or with
    none, and an ordinary call right after is right.  One (chunk, head) a CTA, more of them than SMs, three tiles of columns, small states."""
    from lucciola_b200 import ops
    from lucciola_b200.csrc import library
    if hold in (2, 4) and dim <= 64:
        pytest.skip("the walk on the ordinary pipes, which waits for nothing")
    torch.manual_seed(19)
    lens = [250]
    o, step = gentle(kind, 250, heads, heads, dim, vdim), step_of([250], [0])
    state = 0.3 * torch.randn(1, heads, dim, vdim, device=DEV)
    want, S = plain(kind, o, state, step, heads, heads, dim, vdim)
    fn, real = library().lb_chunk_recurrence_wait_test, ops._call
    fn.argtypes, fn.restype = ops._SIGNATURES["lb_chunk_recurrence"] + [ctypes.c_int, ctypes.c_ulonglong], ctypes.c_int
    held = []

    def call(name, *args):
        if name != "lb_chunk_recurrence":
            return real(name, *args)
        held.append(fn(*args, hold, 200_000))
    assert ops.device_error() == 0
    monkeypatch.setattr(ops, "_call", call)
    kept = state.clone()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    got = through_ops(kind, o, kept, step, heads, heads, dim, vdim, True, shifted=False)
    torch.cuda.synchronize()
    assert time.perf_counter() - t0 < 1.0                # its limit, not the ordinary two seconds
    monkeypatch.setattr(ops, "_call", real)
    assert held == [0]
    assert code <= ops.device_error() < code + 40 and ops.device_error() == 0
    if hold >= 8:
        assert torch.isnan(got).all()
    if hold in (2, 4):
        assert torch.equal(kept, state)
    got = through_ops(kind, o, state, step, heads, heads, dim, vdim, True, shifted=False)
    assert (got.double() - want).abs().max() <= 1e-5 * want.abs().max() and (state.double() - S).abs().max() <= 1e-5 * S.abs().max()
    assert ops.device_error() == 0


# a token by itself, and one, two, four and eight tokens a thread
@pytest.mark.parametrize("tokens,channels", [(1, 64), (8, 64), (3000, 64), (4096, 260), (1200, 1024), (1557, 4096)])
def test_silu_of_the_short_convolution(tokens, channels):
    """Where the activation changes from the reciprocal to the division (80), around the largest and smallest results and at what is no
    number, alone and four in a word, for every number of tokens a thread: x / (1 + e^-x) within two units in the last place for the
    exponential, one half for the sum and one half for the quotient, 3.6e-7, and 3e-37 where the exponential is infinite in 32 bits
    (from -88.7 on)."""
    from lucciola_b200 import ops
    v = [0.0, -0.0, 1e-30, -1e-38, 79.99, -79.99, 80.0, -80.0, 87.0, -87.5, -88.5, -103.0, -200.0, 200.0, 3e38, -3e38, float("inf"), float("-inf"), float("nan"), -1.2785, 0.5]
    x = torch.linspace(-90, 90, tokens * channels, device=DEV).view(tokens, channels)
    x[0, : len(v)] = torch.tensor(v, device=DEV)
    w = torch.zeros(4, channels, device=DEV)
    w[3] = 1
    step, s = step_of([tokens], [0]), torch.cuda.current_stream().cuda_stream
    step.token_seq = torch.zeros(tokens, dtype=torch.int32, device=DEV)
    out = torch.empty_like(x)
    ops.short_conv(out, x, w, None, torch.zeros(1, 3, channels, device=DEV), step, s)
    X = x.double()
    want = X / (1 + torch.exp(-X))
    ok = torch.ones_like(x, dtype=torch.bool)
    ok[:4] = torch.isfinite(x[0])                # a tap of nothing times what is no number is no number in the three tokens behind it
    assert ((out.double() - want).abs()[ok] <= 3.6e-7 * want.abs()[ok] + 3e-37).all()
    inf = float("inf")
    assert out[0, v.index(inf)] == inf and out[0, v.index(-inf)].isnan() and out[0, 18].isnan()
