"""Kernels that are queued behind one another and so start while the one before them still writes what they read: behind the product
that makes their input, the same buffer every time, they must give what they give when each launch is waited for (GPU)."""
import pytest
import torch

from test_chunk_recurrence_gpu import DEV, step_of

pytestmark = pytest.mark.gpu


# rows of one, two, four and eight tokens a thread, of four bytes at a time, and a token a sequence
@pytest.mark.parametrize("channels,lens,shift", [(64, [30, 7], 0), (64, [3000], 0), (2560, [700, 1, 457], 0), (8192, [15, 30, 45, 60, 75, 93], 0), (4096, [1205, 5, 847], 0),
                                                 (2560, [300, 40], 1), (4096, [1] * 300, 0), (4096, [1] * 300, 1)])
def test_short_convolution_behind_its_product(channels, lens, shift):
    from lucciola_b200 import ops
    torch.manual_seed(len(lens) + channels)
    T, s, passes = sum(lens), torch.cuda.current_stream().cuda_stream, 6
    step = step_of(lens, list(range(len(lens))))
    step.token_seq = torch.tensor([i for i, n in enumerate(lens) for _ in range(n)], dtype=torch.int32, device=DEV)
    w = torch.randn(channels + 16, 512, device=DEV).bfloat16()
    x = [torch.randn(T, 512, device=DEV).bfloat16() for _ in range(passes)]
    taps, bias = torch.randn(4, channels, device=DEV), torch.randn(channels, device=DEV)
    busy = torch.randn(4096, 4096, device=DEV)

    def run(wait):
        pre, got = torch.empty(T, channels + 16, device=DEV), []
        state = torch.zeros(len(lens), 3, channels, device=DEV)
        torch.cuda.synchronize()
        done = torch.cuda.synchronize if wait else (lambda: None)
        if not wait:
            busy @ busy                                  # the launches below are all queued before the first of them starts
        for i in range(passes):
            out, at = torch.empty(T, channels, device=DEV), pre[:, 8 + shift:8 + shift + channels]
            ops.gemm_tcgen05(pre, x[i], w, s)
            done()
            if not ops.short_conv_step(out, at, taps, bias, state, step, s):
                ops.short_conv(out, at, taps, bias, state, step, s)
                done()
                ops.short_conv_state(state, at, 4, step, s)
            done()
            got.append(out)
        torch.cuda.synchronize()
        return got + [state]

    want = run(True)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(run(False), want))


def readers():
    from lucciola_b200 import ops
    n, eps = 2048, 1e-6
    w, ones = torch.rand(n, device=DEV), torch.ones(1200, n, device=DEV)
    return {"gated activation": lambda out, p, s: ops.swiglu(out, p[:, :n], p[:, n:2 * n], s),
            "activation": lambda out, p, s: ops.activation(out, p[:, :n], "silu", s),
            "rounded columns": lambda out, p, s: ops.round_cols(out, p[:, 8:8 + n], s),
            "gated group norm": lambda out, p, s: ops.gated_group_norm(out, p[:, :n], p[:, n:2 * n], w, 16, eps, s),
            "gated norm": lambda out, p, s: ops.rmsnorm_gated(out, ones[:p.shape[0]], w, p[:, n:2 * n], 1.0, eps, s)}


@pytest.mark.parametrize("name", ["gated activation", "activation", "rounded columns", "gated group norm", "gated norm"])
@pytest.mark.parametrize("T", [3, 300, 1200])
def test_readers_of_a_product(name, T):
    from lucciola_b200 import ops
    torch.manual_seed(T)
    s, call, passes = torch.cuda.current_stream().cuda_stream, readers()[name], 6
    w = torch.randn(4096 + 16, 512, device=DEV).bfloat16()
    x = [torch.randn(T, 512, device=DEV).bfloat16() for _ in range(passes)]
    busy = torch.randn(4096, 4096, device=DEV)

    def run(wait):
        pre = torch.empty(T, 4096 + 16, device=DEV)
        got = [torch.empty(T, 2048, device=DEV, dtype=torch.float32 if name in ("gated activation", "activation") else torch.bfloat16) for _ in range(passes)]
        torch.cuda.synchronize()
        if not wait:
            busy @ busy
        for i in range(passes):
            ops.gemm_tcgen05(pre, x[i], w, s)
            if wait:
                torch.cuda.synchronize()
            call(got[i], pre, s)
        torch.cuda.synchronize()
        return got

    want = run(True)
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(run(False), want))
