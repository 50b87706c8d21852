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
