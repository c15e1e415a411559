"""Outputs that overlap an input: nothing after the spectrum reads the caller's arrays,
so the result is that of separate buffers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
LAM, DX = 0.6328, 10.0


def _inputs(ph, cuda, nx, ny):
    g = torch.Generator(device=cuda)
    g.manual_seed(nx + ny)
    wf = torch.randn((ny, nx), dtype=torch.complex64, generator=g, device=cuda)
    d = ph.cu_transfer_sqrt_arr(nx, LAM, DX, n_slow=ny)
    return [wf, ph.cu_transfer(-1000.0, nx, LAM, d).data, ph.cu_transfer(-200.0, nx, LAM, d).data]


@pytest.mark.parametrize("nx,ny", [(64, 64), (256, 256), (384, 128), (64, 512)])
@pytest.mark.parametrize("over", [0, 1, 2])
def test_packed_words_over_an_input(ph, cuda, nx, ny, over):
    from ph_gb300 import parallel
    arrays = _inputs(ph, cuda, nx, ny)
    wrap = lambda a: (ph.CuWavefront(a[0]), ph.CuTransfer(a[1]), ph.CuTransfer(a[2]))
    want = parallel.reconst_xyprojection_range(*wrap(arrays), 3, 12)
    inside = [a.clone() for a in arrays]
    packed = inside[over].view(torch.int64)     # 8 bytes per pixel, as the field
    got = parallel.reconst_xyprojection_range(*wrap(inside), 3, 12, packed=packed)
    assert got.data_ptr() == inside[over].data_ptr()
    assert torch.equal(got, want)


@pytest.mark.parametrize("nx,ny", [(64, 64), (256, 256), (384, 128)])
@pytest.mark.parametrize("over", [0, 1, 2])
@pytest.mark.parametrize("shift", [0, 4])
def test_projection_over_an_input(ph, cuda, nx, ny, over, shift):
    """proj inside the input's buffer, at its start and one element on."""
    from ph_gb300 import holofunc
    arrays = _inputs(ph, cuda, nx, ny)
    call = lambda proj, a: ctx.call("ph_reconst_xyproj", proj, None, a[0].data_ptr(), a[1].data_ptr(), a[2].data_ptr(),
                                    nx, ny, 9, s)
    ctx, s = holofunc._ctx_stream(arrays[0])
    want = torch.empty((ny, nx), dtype=torch.float32, device=cuda)
    call(want.data_ptr(), arrays)
    inside = [a.clone() for a in arrays]
    call(inside[over].data_ptr() + shift, inside)
    got = inside[over].view(torch.float32).reshape(-1)[shift // 4: shift // 4 + nx * ny].reshape(ny, nx)
    assert torch.equal(got, want)
