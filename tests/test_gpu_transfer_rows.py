"""The transfer that propagation forms on the way (a fixed-point phase, FP64 outside its
range), value by value: it is the spectrum of a propagated point."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
LAM = 0.6328


def _spectrum(ph, cuda, d, z):
    n = d.shape[0]
    point = torch.zeros((n, n), dtype=torch.complex64, device=cuda)
    point[0, 0] = 1.0                      # every coefficient is one, exactly
    out = ph.CuWavefront(torch.empty_like(point))
    ph.cu_asm_prop_(out, ph.CuWavefront(point), ph.CuTransferSqrtPart(torch.from_numpy(d).to(cuda)), z, n, LAM)
    return np.fft.fftshift(np.fft.fft2(out.data.cpu().numpy().astype(np.complex128)))


@pytest.mark.parametrize("n", [128, 256, 1024])
# (the last lies beyond |z / lambda| = 2^40; below it, where FP64 rounds the phase by less than 1e-7)
@pytest.mark.parametrize("z", [0.0, 1e-9, -5000.0, 80000.0, 5.0e7, 7.0e11])
def test_each_value(ph, cuda, n, z):
    rng = np.random.default_rng(n)
    d = rng.uniform(0.0, 1.0, (n, n)).astype(np.float32)
    s = np.array([1.0, 1.0 - 2.0 ** -24, 0.5, 0.5 + 2.0 ** -24, 2.0 ** -15, 2.0 ** -30, 2.0 ** -30 - 2.0 ** -54, 2.0 ** -31,
                  1.0 + 2.0 ** -23, 1.5, 2.0, 0.0])
    d.reshape(-1)[:12] = s * s             # the range's ends, mantissas of all ones and of none
    d.reshape(-1)[12:16] = [1e-19, 1e-30, 1e-38, 4.0]
    phase = (2.0 * np.pi * z) / LAM * np.sqrt(d).astype(np.float64)
    off = np.abs(_spectrum(ph, cuda, d, z) - np.exp(1j * phase))
    # The inverse transform's noise, 2e-7 in relative L2, is spread evenly over the spectrum:
    # about 1.4e-7 per component, six times that at most.  A wrong value would stand out.
    assert off.max() <= 1.2e-6


@pytest.mark.parametrize("bad", [np.nan, -1.0])
def test_no_value(ph, cuda, bad):
    d = np.full((128, 128), 0.5, np.float32)
    d[3, 5] = bad
    assert np.isnan(_spectrum(ph, cuda, d, 1000.0)).all()
