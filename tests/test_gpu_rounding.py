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
