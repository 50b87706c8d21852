"""Which form of a recurrence a step takes, by the lengths of its portions (CPU: the rule alone)."""
from types import SimpleNamespace

import pytest

KINDS = ["fixed", "ssm", "hgrn2", "delta", "channels"]


def portions(kind, lens, heads=16, dim=128, vdim=128):
    from lucciola_b200 import ops
    return ops.chunk_portions(kind, SimpleNamespace(num_seqs=len(lens), q_lens=list(lens), max_q_len=max(lens)), heads, dim, vdim)


@pytest.mark.parametrize("kind", KINDS)
def test_a_step_goes_as_a_whole(kind):
    """Beside a portion that pays for the launches every portion of 32 tokens goes with it, and only shorter ones stay behind."""
    assert portions(kind, [2048]) == ([0], 32)
    assert portions(kind, [105, 2048, 31, 32, 1]) == ([0, 1, 3], 32)
    assert portions(kind, [1] * 32 + [700]) == ([32], 32)
    assert portions(kind, [31] * 9) == ([], 0) and portions(kind, [40]) == ([], 0) and portions(kind, [1] * 64) == ([], 0)


# portions (16 heads of 128 x 128; state space 32 of 128 x 64) and the us of both forms, all launches: token by token | chunked
@pytest.mark.parametrize("kind,lens,walk,chunk", [
    ("fixed", [96], 21, 58), ("fixed", [448], 98, 64), ("fixed", [160] * 3, 90, 67), ("fixed", [64] * 3, 39, 54), ("fixed", [128] * 16, 269, 160),
    ("ssm", [96], 26, 35), ("ssm", [256], 63, 40), ("ssm", [96] * 16, 138, 153), ("ssm", [448] * 5, 237, 153), ("ssm", [48] * 3, 23, 40),
    ("hgrn2", [192], 41, 63), ("hgrn2", [448], 91, 70), ("hgrn2", [128] * 3, 57, 71), ("hgrn2", [320] * 3, 132, 76), ("hgrn2", [224] * 5, 141, 117),
    ("delta", [96], 46, 69), ("delta", [256], 114, 72), ("delta", [64] * 5, 66, 74), ("delta", [65] * 16, 151, 202), ("delta", [224] * 8, 240, 206),
    ("channels", [128], 62, 93), ("channels", [320], 146, 103), ("channels", [96] * 3, 66, 86), ("channels", [256] * 3, 160, 131), ("channels", [96] * 16, 298, 260)])
def test_the_faster_form(kind, lens, walk, chunk):
    heads, dim, vdim = (32, 128, 64) if kind == "ssm" else (16, 128, 128)
    assert bool(portions(kind, lens, heads, dim, vdim)[0]) == (chunk < walk)


def test_single_tokens_of_small_states_are_walked():
    from lucciola_b200 import ops
    state = SimpleNamespace(data_ptr=lambda: 4096)
    one = lambda lens, dim, vdim: ops.single_tokens(SimpleNamespace(num_seqs=len(lens), q_lens=lens, max_q_len=max(lens)), dim, vdim, state)
    assert one([1], 64, 64) and one([1] * 200, 128, 68)
    assert not one([1], 63, 64) and not one([1], 64, 60) and not one([1], 129, 64) and not one([1], 64, 66) and not one([1, 2], 64, 64)


def test_what_the_kernels_do_not_take():
    assert portions("delta", [9999], dim=129) == ([], 0)                    # more rows of the state than the kernels hold
    assert portions("delta", [9999], vdim=5000) == ([], 0)
    from lucciola_b200 import ops
    assert ops.chunk_portions("delta", SimpleNamespace(num_seqs=3, q_lens=[], max_q_len=9999), 2, 64, 64) == ([], 0)      # lengths the host does not know
