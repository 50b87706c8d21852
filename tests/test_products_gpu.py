"""Products on the tensor cores where one kernel, tile or store gives way to another: token counts and ratios of features to places
on both sides of every line, rows that begin on 32-, 16- and 2-byte boundaries, and inner sizes that end inside a stage of a ring
of any length, against the product in 64 bits (GPU)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def check(M, N, K, dtype, ldy, shift, force_bt=0, force_splits=0):
    from lucciola_b200 import ops
    torch.manual_seed(M * 7 + N + K)
    x = torch.randn(M, K, device=DEV).bfloat16()
    w = torch.randn(N, K, device=DEV).bfloat16()
    whole = torch.full((M, ldy), 7.0, device=DEV, dtype=dtype)
    y = whole[:, shift:shift + N]
    ops.gemm_tcgen05(y, x, w, torch.cuda.current_stream().cuda_stream, force_bt=force_bt, force_splits=force_splits)
    want = x.double() @ w.double().T
    # sums of K products of 8-bit numbers: the accumulator drops less than 2^-22 of the largest partial sum each 16 places, the output rounds once
    bound = K / 16 * 2.0 ** -22 * (x.double().abs() @ w.double().abs().T) + (2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -23) * want.abs()
    assert ((y.double() - want).abs() <= bound + 1e-30).all()
    rest = torch.cat([whole[:, :shift], whole[:, shift + N:]], dim=1)
    assert (rest == 7.0).all(), "written outside the product's columns"


@pytest.mark.parametrize("M", [32, 33, 64, 65, 128, 129, 256, 257])
@pytest.mark.parametrize("N,K", [(384, 256), (376, 256), (256, 256), (248, 256), (128, 256), (120, 256), (2048, 2048), (2176, 2048), (264, 2056)])
def test_on_both_sides_of_every_line(M, N, K):
    check(M, N, K, torch.bfloat16, N, 0)


@pytest.mark.parametrize("M", [59, 93, 128, 200])
@pytest.mark.parametrize("N,K", [(12288, 4096), (4096, 4096), (2048, 4096)])
def test_32_bit_sums_in_short_chains(M, N, K):
    """32-bit outputs of up to 256 tokens are no further from 64 bits than with the kernel that cuts K over a cluster and the cut that
    it takes by itself (a quarter more than that for another order of the same sums); with more features than places from 129 tokens on, one
    chain, which the bound of `check` holds."""
    from lucciola_b200 import ops
    torch.manual_seed(M + N)
    x, w, s = torch.randn(M, K, device=DEV).bfloat16(), torch.randn(N, K, device=DEV).bfloat16(), torch.cuda.current_stream().cuda_stream
    want = x.double() @ w.double().T
    def off(**kw):
        y = torch.empty(M, N, device=DEV)
        ops.gemm_tcgen05(y, x, w, s, **kw)
        return ((y.double() - want) ** 2).mean().sqrt()
    if M > 128 and N > K:
        check(M, N, K, torch.float32, N, 0)
    else:
        assert off() <= 1.25 * off(force_bt=128 if M > 64 else 64)


def plan(M, N, K):
    """(splits, token tile) of the kernel that cuts K over a cluster."""
    import ctypes
    from lucciola_b200.csrc import library
    bt = ctypes.c_int()
    f = library().lb_gemm_tcgen05_plan
    f.argtypes, f.restype = [ctypes.c_int] * 3 + [ctypes.c_void_p], ctypes.c_int
    return f(M, N, K, ctypes.addressof(bt)), bt.value


def as_the_cluster_adds(M, N, K, dtype, swiglu=False):
    """Whichever kernel takes it: the bits of the kernel that cuts K over a cluster, as many ranges as it takes by itself, with rows that lack
    their norm's factor (17 partial sums a row: more than one round of the loads that add them up), and without, and with an element operation."""
    from lucciola_b200 import ops
    torch.manual_seed(M + N + K)
    x, w, s = torch.randn(M, K, device=DEV).bfloat16(), torch.randn(N, K, device=DEV).bfloat16(), torch.cuda.current_stream().cuda_stream
    splits, bt = plan(M, N, K)
    sumsq = K / 17 * (0.5 + torch.rand(M, 17, device=DEV))
    for kw in (dict(), dict(sumsq=sumsq, eps=1e-6)) + (() if swiglu else (dict(post="gelu"),)):
        got, want = (torch.empty(M, N // 2 if swiglu else N, device=DEV, dtype=dtype) for _ in range(2))
        ops.gemm_tcgen05(got, x, w, s, swiglu=swiglu, **kw)
        ops.gemm_tcgen05(want, x, w, s, swiglu=swiglu, force_bt=bt, force_splits=splits, **kw)
        assert torch.equal(got, want), kw
    assert ops.device_error() == 0
    return splits


# features and places, and the splits of 33 to 128 | 129 to 256 tokens, on both sides of the lines; widths that are no multiple of a tile, and sums
# that fill tensor memory (eight of 64 columns)
@pytest.mark.parametrize("M", [33, 64, 65, 93, 128, 129, 200, 256])
@pytest.mark.parametrize("N,K,splits", [(4096, 2048, (8, 4)), (2048, 2048, (8, 8)), (2600, 2056, (8, 6)), (3000, 4104, (8, 5)), (4800, 3200, (6, 3)), (6144, 4096, (5, 2)),
                                        (8192, 4096, (4, 2)), (4100, 4104, (7, 3)), (1000, 2000, (8, 8)), (12288, 4096, (2, 1)), (17000, 2048, (2, 1)), (600, 384, (1, 1)),
                                        (1600, 1032, (4, 4))])
def test_16_bit_sums_keep_the_cut(M, N, K, splits):
    if M > 128 and N > K:
        pytest.skip("one chain")
    assert as_the_cluster_adds(M, N, K, torch.bfloat16) == splits[M > 128]


@pytest.mark.parametrize("M", [1, 7, 8, 16, 17, 32])
@pytest.mark.parametrize("N,K", [(12288, 2048), (12289, 512), (12288, 2056), (16384, 3064), (16384, 3072), (18816, 1024)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_few_tokens_of_many_features(M, N, K, dtype):
    """Two splits, by two CTAs or, on the one side of the lines in tokens, places and types, by one."""
    assert as_the_cluster_adds(M, N, K, dtype) == 2
    check(M, N, K, dtype, N, 0)
    if N % 128 == 0:
        assert as_the_cluster_adds(M, N, K, dtype, swiglu=True) == 2


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("ldy,shift", [(320, 0), (328, 8), (324, 4), (321, 1), (336, 16)])
@pytest.mark.parametrize("M", [130, 300, 1100])
def test_rows_on_any_boundary(M, ldy, shift, dtype):
    check(M, 300, 136, dtype, ldy, shift, force_bt=-1)


@pytest.mark.parametrize("width", [16, 64, 96, 128, 160, 256])
@pytest.mark.parametrize("K", [8, 64, 72, 520, 1032])
@pytest.mark.parametrize("pairs", [False, True])
def test_rings_of_any_length(width, K, pairs):
    if pairs and width % 32:
        pytest.skip("pairs take widths that are multiples of 32")
    check(300, 1000, K, torch.float32, 1000, 0, force_bt=-2 if pairs else -1, force_splits=width)
