"""Rounding of the two-stage passes, against counts of the roundings they need.

One FP32 rounding of a component in [1/2, 1) is off by 2^-24 / sqrt(12) in the root mean
square (spacing 2^-24), 1.7e-8; a complex product rounds each component twice."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
LAM, DX = 0.6328, 10.0
ROUNDING = 2.0 ** -24 / np.sqrt(12.0)


@pytest.mark.parametrize("ny", [128, 256, 768, 1024, 1536, 2048, 4096])
def test_slices_of_a_uniform_field(ph, cuda, ny):
    """A uniform field has one coefficient, whose slices are hf hdz^k.  The chain of
    products may add their own roundings only: those of the step itself would add up (and
    every pixel of a hologram shows this coefficient's error)."""
    nx, slices = 128, 16
    d = ph.cu_transfer_sqrt_arr(nx, LAM, DX, n_slow=ny)
    wave = ph.CuWavefront(torch.ones((ny, nx), dtype=torch.complex64, device=cuda))
    off = []
    for dz in np.linspace(50.0, 500.0, 24):
        tf, td = ph.cu_transfer(-5000.0, nx, LAM, d), ph.cu_transfer(-float(dz), nx, LAM, d)
        got = ph.cu_get_reconst_complex_vol(wave, tf, td, slices).to(torch.complex128).mean((1, 2)).cpu().numpy()
        front, step = (complex(t.data[ny // 2, nx // 2].item()) for t in (tf, td))
        want = front * step ** np.arange(slices)
        off.append(np.abs(got - want) / np.abs(want))
    # 2 components x 2 roundings per product; 7.5 products of the chain on average, and four
    # more for the first slice's phase, modulus, rotation and scale; half as much again
    assert np.sqrt(np.mean(np.square(off))) <= 1.5 * ROUNDING * np.sqrt(2 * 2 * (7.5 + 4))


def test_propagation_by_nothing(ph, cuda):
    """White noise through two transforms each way at 128 = 8 x 16, with a transfer of one.
    Per transform: 7 levels of additions at 2.75e-8 each (a rounding over the spread of
    mantissas), and 1.75 twiddle products (the stage's, half of radix 16's and a quarter of
    radix 8's are not trivial) of 4.4e-8: the factor's rounding and the product's two.
    1.86e-7 in all; stage twiddles formed as products of two rounded factors make it 2.04e-7."""
    n = 128
    g = torch.Generator(device=cuda)
    g.manual_seed(128)
    u = torch.randn((n, n), dtype=torch.complex64, generator=g, device=cuda)
    out = ph.CuWavefront(torch.empty_like(u))
    one = ph.CuTransferSqrtPart(torch.ones((n, n), dtype=torch.float32, device=cuda))
    ph.cu_asm_prop_(out, ph.CuWavefront(u), one, 0.0, n, LAM)
    off = (out.data.to(torch.complex128) - u).abs().square().sum() / u.to(torch.complex128).abs().square().sum()
    assert float(off.sqrt()) <= 1.95e-7


@pytest.mark.parametrize("n", [128, 192, 256, 384, 512, 768, 1024, 1536, 2048, 3072, 4096])
def test_transforms_keep_the_modulus(ph, cuda, n):
    """The part of the error that is a common factor.  1 / sqrt(2) and sqrt(3) / 2 round to
    less by 1.7e-8, and shrink a field by up to 1.5e-7 in two transforms there and two back
    unless the stage twiddles make up for it; of these a quarter may be left."""
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    u = torch.randn((n, n), dtype=torch.complex64, generator=g, device=cuda)
    out = ph.CuWavefront(torch.empty_like(u))
    one = ph.CuTransferSqrtPart(torch.ones((n, n), dtype=torch.float32, device=cuda))
    ph.cu_asm_prop_(out, ph.CuWavefront(u), one, 0.0, n, LAM)
    u = u.to(torch.complex128)
    factor = float((out.data.to(torch.complex128) * u.conj()).sum().real / u.abs().square().sum())
    scale = float(np.float32(1.0 / n ** 2)) * n ** 2     # 1 / n^2 is rounded where n has a factor of three
    assert abs(factor / scale - 1.0) <= 4e-8
