"""The transfer function against FP64: both signs and magnitudes of the distance, and
square-root terms outside the range of propagation's fixed-point phase."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
LAM = 0.6328
ULP = 2.0 ** -24   # spacing of Float32 in [1/2, 1): both sides round the exact value once


@pytest.mark.parametrize("n,z", [(1, 80000.0), (3, -5000.0), (5, 1.0e9), (50, 123456.7), (64, -200.0), (64, 0.0),
                                 (64, 1e-9), (250, 5000.0), (1024, -200000.0)])
def test_transfer_matches_fp64(ph, cuda, n, z):
    rng = np.random.default_rng(n)
    d = rng.uniform(0.0, 1.0, (n, n)).astype(np.float32)
    d.reshape(-1)[: min(n * n, 4)] = [1.0, 0.0, 1e-19, 1e-30][: min(n * n, 4)]
    got = ph.cu_transfer(z, n, LAM, ph.CuTransferSqrtPart(torch.from_numpy(d).to(cuda))).data.cpu().numpy()
    phase = (2.0 * np.pi * z) / LAM * np.sqrt(d).astype(np.float64)
    # the reference's own phase is rounded to FP64: at |phase| = 1e10 that is 1e-6 rad
    tol = ULP * 1.01 + np.abs(phase).max() * 2.0 ** -52
    assert np.abs(got.real - np.cos(phase)).max() <= tol
    assert np.abs(got.imag - np.sin(phase)).max() <= tol


def test_values_outside_the_range(ph, cuda):
    d = np.array([[np.nan, -1.0], [4.0, 1.5]], np.float32)
    got = ph.cu_transfer(1000.0, 2, LAM, ph.CuTransferSqrtPart(torch.from_numpy(d).to(cuda))).data.cpu().numpy()
    assert np.isnan(got[0].real).all() and np.isnan(got[0].imag).all()
    phase = (2.0 * np.pi * 1000.0) / LAM * np.sqrt(d[1]).astype(np.float64)
    assert np.abs(got[1] - np.exp(1j * phase)).max() <= 2 * ULP


@pytest.mark.parametrize("n,z", [(128, 80000.0), (128, -5000.0), (192, 1.0e9), (256, 1e-9), (1024, -200000.0)])
def test_propagation_forms_the_same_transfer(ph, cuda, n, z):
    """The spectrum of a propagated point is the transfer (centred); its values pass one
    forward and one inverse Float32 transform, 1e-6 in relative L2."""
    rng = np.random.default_rng(n)
    d = rng.uniform(0.0, 1.0, (n, n)).astype(np.float32)
    d.reshape(-1)[:6] = [1.0, 0.0, 1e-19, 1e-30, 1.5, 4.0]
    point = torch.zeros((n, n), dtype=torch.complex64, device=cuda)
    point[0, 0] = 1.0
    out = ph.CuWavefront(torch.empty_like(point))
    ph.cu_asm_prop_(out, ph.CuWavefront(point), ph.CuTransferSqrtPart(torch.from_numpy(d).to(cuda)), z, n, LAM)
    got = np.fft.fftshift(np.fft.fft2(out.data.cpu().numpy().astype(np.complex128)))
    phase = (2.0 * np.pi * z) / LAM * np.sqrt(d).astype(np.float64)
    ref = np.exp(1j * phase)
    tol = 1e-6 + np.abs(phase).max() * 2.0 ** -52
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) <= tol
