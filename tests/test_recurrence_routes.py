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


# portions (16 heads of 128 x 128; state space 32 of 128 x 64) and the us of both forms, all launches: token by token | chunked.  The first of the
# lines that begin with 97 and 193 tokens, and both sides of the 148 (chunk, head)s that run at once (560 and 600 tokens).
@pytest.mark.parametrize("kind,lens,walk,chunk", [
    ("fixed", [96], 22, 24), ("fixed", [160], 36, 24), ("fixed", [448], 98, 30), ("fixed", [560], 122, 31), ("fixed", [600], 131, 38), ("fixed", [97] * 3, 59, 32),
    ("fixed", [160] * 3, 89, 32), ("fixed", [96] * 9, 108, 53), ("fixed", [128] * 16, 269, 105),
    ("ssm", [97], 27, 22), ("ssm", [256], 65, 25), ("ssm", [48] * 3, 23, 27), ("ssm", [128] * 3, 51, 36), ("ssm", [97] * 9, 78, 81), ("ssm", [96] * 16, 139, 145),
    ("ssm", [448] * 5, 239, 147),
    ("hgrn2", [96], 22, 30), ("hgrn2", [193], 42, 31), ("hgrn2", [448], 90, 36), ("hgrn2", [560], 112, 37), ("hgrn2", [600], 121, 52), ("hgrn2", [64] * 3, 31, 33),
    ("hgrn2", [193] * 3, 85, 56), ("hgrn2", [320] * 3, 131, 60), ("hgrn2", [224] * 5, 140, 95),
    ("delta", [80], 40, 41), ("delta", [112], 54, 41), ("delta", [256], 115, 48), ("delta", [560], 244, 65), ("delta", [600], 262, 76), ("delta", [97] * 3, 61, 66),
    ("delta", [128] * 3, 77, 66), ("delta", [65] * 16, 150, 191), ("delta", [224] * 8, 240, 197),
    ("channels", [128], 61, 69), ("channels", [160], 75, 61), ("channels", [320], 142, 67), ("channels", [560], 245, 82), ("channels", [600], 262, 110),
    ("channels", [97] * 3, 67, 77), ("channels", [256] * 3, 160, 131), ("channels", [96] * 16, 300, 270)])
def test_the_faster_form(kind, lens, walk, chunk):
    heads, dim, vdim = (32, 128, 64) if kind == "ssm" else (16, 128, 128)
    assert bool(portions(kind, lens, heads, dim, vdim)[0]) == (chunk < walk)


@pytest.mark.parametrize("kind,lens,walk,chunk", [
    ("fixed", [64] * 3, 38, 27), ("fixed", [80] * 32, 323, 185), ("ssm", [96], 26, 23), ("ssm", [96] * 3, 40, 36), ("hgrn2", [192], 40, 31), ("hgrn2", [180] * 3, 79, 38),
    ("hgrn2", [96] * 4, 44, 38), ("delta", [96], 46, 41), ("delta", [64] * 9, 81, 71), ("channels", [96] * 4, 105, 79)])
def test_short_portions_stay_where_they_were(kind, lens, walk, chunk):
    """Below 97 tokens (HGRN2 193) the times of the kernels before decide: these steps are walked, although the chunked form would be the faster."""
    heads, dim, vdim = (32, 128, 64) if kind == "ssm" else (16, 128, 128)
    assert chunk < walk and portions(kind, lens, heads, dim, vdim) == ([], 0)


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
