"""Calls at the limits of a context's scratch: after ph_reserve under a stream capture, and
with a budget that holds the smallest form of a call only."""
import pytest
import torch

pytestmark = pytest.mark.gpu
LAM, DX = 0.6328, 10.0


def _retrieval(ph, cuda, n):
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    h1, h2 = (0.1 + torch.rand((n, n), generator=g, device=cuda) for _ in range(2))
    d = ph.cu_transfer_sqrt_arr(n, LAM, DX)
    return h1, h2, ph.cu_transfer(700.0, n, LAM, d).data, ph.cu_transfer(-700.0, n, LAM, d).data


def _call(ctx, out, arrays, n, iters=2):
    s = torch.cuda.current_stream().cuda_stream
    ctx.call("ph_phase_retrieval", out.data_ptr(), *(a.data_ptr() for a in arrays), n, n, iters, None, s)


@pytest.mark.parametrize("n", [64, 128, 192, 256, 768])
def test_retrieval_captured_after_reserve(ph, cuda, n):
    """ph_reserve for one slice, then a captured retrieval; a call outside the capture does
    not move the scratch that the graph holds."""
    from ph_gb300 import _lib
    arrays = _retrieval(ph, cuda, n)
    want, out = (torch.zeros((n, n), dtype=torch.complex64, device=cuda) for _ in range(2))
    _call(_lib.default_context(0), want, arrays, n)
    ctx = _lib.Context(0)
    ctx.call("ph_reserve", n, n, 1, torch.cuda.current_stream().cuda_stream)
    held = ctx.scratch_bytes
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _call(ctx, out, arrays, n)
    again = torch.zeros_like(out)
    _call(ctx, again, arrays, n)
    assert ctx.scratch_bytes == held
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and torch.equal(again, want)
    del graph


@pytest.mark.parametrize("n", [128, 192, 512])
@pytest.mark.parametrize("reserve", [False, True])
def test_retrieval_in_the_smallest_budget(ph, cuda, n, reserve):
    """16 bytes per pixel hold the one-shot passes; the other forms take 40."""
    from ph_gb300 import _lib
    arrays = _retrieval(ph, cuda, n)
    want, out = (torch.zeros((n, n), dtype=torch.complex64, device=cuda) for _ in range(2))
    _call(_lib.default_context(0), want, arrays, n)
    ctx = _lib.Context(0, hbm_budget_bytes=(33 if reserve else 16) * n * n + 1024)
    if reserve:   # 32 bytes per pixel for a slice, and its accumulators
        ctx.call("ph_reserve", n, n, 1, torch.cuda.current_stream().cuda_stream)
    _call(ctx, out, arrays, n)
    assert ctx.scratch_bytes <= (33 if reserve else 16) * n * n + 1024
    assert float((out - want).abs().square().sum().sqrt() / want.abs().square().sum().sqrt()) < 4e-5
