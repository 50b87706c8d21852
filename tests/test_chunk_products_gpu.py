"""The chunked recurrences where their products' tiles, rings and CTAs change over: value columns in one tile of 64, of 128 and in several,
more (chunk, head)s than SMs, so that a CTA takes several one behind the other, and a value that is not finite behind the first
tile of columns; against the plain recurrence in 64 bits (GPU)."""
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
